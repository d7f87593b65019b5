// Pinned host memory: ordinary anonymous memory, in huge pages where it is
// large enough, page-locked once its pages are there.
//
// What bounds a new block is its pages: the kernel clears them one by one, and
// the driver looks each one up to lock it. Huge pages leave a five-hundredth of
// them. A new block and the first copy into it, against the runtime's
// allocation (and, in parentheses, ordinary memory, whose pages come with the
// first copy): 4 MB 1.1 ms, 2.2 (2.0); 8 MB 2.0, 4.1 (3.9); 32 MB 6.8, 13.4
// (15.6). A small block costs 0.3 ms for the locking alone, 64 KB or 1 MB alike
// (0.95 and 1.6 from the runtime), so small blocks are cut from slabs.
//
// Either can take far longer, since the driver serves one memory call at a time
// for all processes on the machine: 20-110 ms now and then, once half a second,
// which a served client saw as the wait for its preview. So programs that
// allocate while chunks run reserve room ahead (host_reserve).
//
// And it is the process's own memory: a forked child has a copy of what was in
// it, where it shares the runtime's with the parent's later results.
#include "host_memory.cuh"

#include <sys/mman.h>

#include <algorithm>
#include <cstdint>
#include <map>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

namespace mcrt {
namespace {

constexpr size_t kPage = 4096;
constexpr size_t kHuge = 2u << 20;
constexpr size_t kSlab = 4u << 20;
constexpr size_t kSlabBlock = kSlab / 2;  // larger blocks are mapped by themselves

// A mapping, page-locked for every device.
struct Mapping {
  char* base = nullptr;
  size_t bytes = 0;
  int device = 0;                 // whose context locked it
  std::map<size_t, size_t> free;  // a slab's free ranges: offset -> length
  size_t used = 0;
  bool reserved = false;
};

struct Block {
  Mapping* in;
  size_t bytes;
};

struct HostMemory {
  std::mutex mu;
  std::map<char*, std::unique_ptr<Mapping>> mappings;
  std::map<char*, Block> blocks;  // handed out
  size_t reserved = 0;            // bytes of the reserved mappings
  int reservations = 0;
};

// Never destroyed: blocks may come back while the process ends.
HostMemory& memory() {
  static HostMemory* m = new HostMemory();
  return *m;
}

cudaError_t map_pinned(size_t bytes, std::unique_ptr<Mapping>* out) {
  auto m = std::make_unique<Mapping>();
  cudaError_t e = cudaGetDevice(&m->device);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return e;
  }
  const size_t align = bytes >= kHuge ? kHuge : kPage;
  const size_t room = bytes + (align - kPage);
  if (room < bytes) return cudaErrorMemoryAllocation;
  void* p = mmap(nullptr, room, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  if (p == MAP_FAILED) return cudaErrorMemoryAllocation;
  char* first = static_cast<char*>(p);
  m->base = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(first) + align - 1) / align * align);
  m->bytes = bytes;
  const size_t before = static_cast<size_t>(m->base - first), after = room - before - bytes;
  if (before) munmap(first, before);
  if (after) munmap(m->base + bytes, after);
  if (align == kHuge) madvise(m->base, bytes, MADV_HUGEPAGE);  // ordinary pages do as well
  for (size_t i = 0; i < bytes; i += kPage) *static_cast<volatile char*>(m->base + i) = 0;
  e = cudaHostRegister(m->base, bytes, cudaHostRegisterPortable);
  if (e != cudaSuccess) {
    cudaGetLastError();  // callers go on without: the next launch's check must not find it
    munmap(m->base, bytes);
    return e;
  }
  *out = std::move(m);
  return cudaSuccess;
}

void unmap_pinned(const Mapping& m) {
  const auto unmap = [&] {
    // Memory that cannot be unlocked (its context is gone) is left.
    if (cudaHostUnregister(m.base) == cudaSuccess) {
      munmap(m.base, m.bytes);
    } else {
      cudaGetLastError();
    }
  };
  int current = -1;
  if (cudaGetDevice(&current) == cudaSuccess && current == m.device) {
    unmap();
    return;
  }
  // A result may be dropped on a thread that works with another device, or with none yet.
  std::thread([&] {
    if (cudaSetDevice(m.device) == cudaSuccess) unmap();
  }).join();
}

// The first free range of a slab that holds `bytes`, or nullptr.
char* cut(Mapping& m, size_t bytes) {
  for (auto it = m.free.begin(); it != m.free.end(); ++it) {
    const size_t at = it->first, length = it->second;
    if (length < bytes) continue;
    m.free.erase(it);
    if (length > bytes) m.free[at + bytes] = length - bytes;
    m.used += bytes;
    return m.base + at;
  }
  return nullptr;
}

void uncut(Mapping& m, char* p, size_t bytes) {
  size_t at = static_cast<size_t>(p - m.base);
  m.used -= bytes;
  auto next = m.free.lower_bound(at);
  if (next != m.free.end() && next->first == at + bytes) {
    bytes += next->second;
    next = m.free.erase(next);
  }
  if (next != m.free.begin()) {
    auto prev = std::prev(next);
    if (prev->first + prev->second == at) {
      at = prev->first;
      bytes += prev->second;
      m.free.erase(prev);
    }
  }
  m.free[at] = bytes;
}

}  // namespace

cudaError_t host_alloc(size_t bytes, void** out) {
  *out = nullptr;
  if (bytes > SIZE_MAX / 2) return cudaErrorMemoryAllocation;
  bytes = (std::max<size_t>(bytes, 1) + kPage - 1) / kPage * kPage;
  HostMemory& h = memory();
  const bool slab = bytes <= kSlabBlock;
  std::unique_ptr<Mapping> made;
  std::unique_lock<std::mutex> lock(h.mu);
  for (auto& m : h.mappings) {
    char* p = cut(*m.second, bytes);
    if (!p) continue;
    h.blocks[p] = Block{m.second.get(), bytes};
    *out = p;
    return cudaSuccess;
  }
  lock.unlock();  // the driver is not waited for under the lock
  const cudaError_t e = map_pinned(slab ? kSlab : bytes, &made);
  if (e != cudaSuccess) return e;
  made->free[0] = made->bytes;
  Mapping* m = made.get();
  char* p = cut(*m, bytes);
  lock.lock();
  h.mappings[m->base] = std::move(made);
  h.blocks[p] = Block{m, bytes};
  *out = p;
  return cudaSuccess;
}

bool host_free(void* pointer) {
  HostMemory& h = memory();
  std::unique_ptr<Mapping> gone;
  {
    std::lock_guard<std::mutex> lock(h.mu);
    const auto it = h.blocks.find(static_cast<char*>(pointer));
    if (it == h.blocks.end()) return false;
    const Block b = it->second;
    uncut(*b.in, it->first, b.bytes);
    h.blocks.erase(it);
    if (b.in->used == 0 && !b.in->reserved) {  // the last block of its mapping
      const auto m = h.mappings.find(b.in->base);
      gone = std::move(m->second);
      h.mappings.erase(m);
    }
  }
  if (gone) unmap_pinned(*gone);
  return true;
}

cudaError_t host_reserve(size_t bytes) {
  if (bytes > SIZE_MAX / 2) return cudaErrorMemoryAllocation;
  bytes = (std::max<size_t>(bytes, 1) + kPage - 1) / kPage * kPage;
  HostMemory& h = memory();
  std::unique_lock<std::mutex> lock(h.mu);
  const size_t have = h.reserved;
  h.reservations++;
  if (have >= bytes) return cudaSuccess;
  h.reserved = bytes;  // another thread's reservation counts on it meanwhile
  lock.unlock();
  std::unique_ptr<Mapping> made;
  const cudaError_t e = map_pinned(bytes - have, &made);
  lock.lock();
  if (e != cudaSuccess) {
    h.reserved -= bytes - have;
    h.reservations--;
    return e;
  }
  made->free[0] = made->bytes;
  made->reserved = true;
  char* base = made->base;
  h.mappings[base] = std::move(made);
  return cudaSuccess;
}

void host_unreserve() {
  HostMemory& h = memory();
  std::vector<std::unique_ptr<Mapping>> gone;
  {
    std::lock_guard<std::mutex> lock(h.mu);
    if (h.reservations == 0 || --h.reservations > 0) return;
    h.reserved = 0;
    for (auto it = h.mappings.begin(); it != h.mappings.end();) {
      Mapping& m = *it->second;
      m.reserved = false;
      if (m.used == 0) {
        gone.push_back(std::move(it->second));
        it = h.mappings.erase(it);
      } else {
        ++it;
      }
    }
  }
  for (const auto& m : gone) unmap_pinned(*m);
}

}  // namespace mcrt
