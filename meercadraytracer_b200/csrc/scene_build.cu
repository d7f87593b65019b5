// GPU binned-SAH BVH build and geometry compile (src/bvh.ts:16-178,
// src/compile.ts:359-432).
//
// The build makes exactly the reference's decisions: per-triangle bounds and
// centroids are computed in double and rounded to float as the reference's
// Float32Array stores do; bins, areas and SAH costs are computed in double;
// this file is compiled without fused multiply-add contraction so every double
// operation rounds as JavaScript's does. Hence every node splits the same set
// of triangles as the reference, with the same 16 bins, leaves of at most 4
// (SAH leaves up to 16) and depth at most 100. Only the numbering of nodes
// (breadth first here) and the order of triangles inside a leaf may differ;
// partitions here are stable.
#include <cuda_runtime.h>

#include <cub/block/block_reduce.cuh>
#include <cub/block/block_scan.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <stdexcept>
#include <string>
#include <vector>

#include "device_scene.cuh"
#include "scene_build.cuh"

namespace mcrt {

namespace {

constexpr int kBins = 16;      // bvh.ts:3 (the default; a build may ask for up to kMaxBins)
constexpr int kMaxBins = 32;
static_assert(kBins <= kMaxBins, "the default bin count must fit the bin arrays");
constexpr int kMaxLeaf = 4;    // bvh.ts:4
constexpr int kBuildDepth = 100;  // bvh.ts:5
constexpr int kBuildBlock = 256;
// A node of at most kTinyMax triangles is finished by one lane (lane_subtree):
// 12 measured best of 6 to 32 (16.4 M triangles rebuilt and traced: 44.8 ms at
// 6, 40.8 at 12, 42.0 at 16, 59.8 at 32).
constexpr int kTinyMax = 12;
// Of nodes of at least kWideMin triangles small children count as a level (BuildCtl::slot_depth).
constexpr int kWideMin = 1 << 15;

void check(cudaError_t e, const char* what) {
  if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}

template <class T>
struct DevArray {
  T* p = nullptr;
  size_t n = 0;
  ~DevArray() { reset(); }
  void reset() {
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
  }
  T* ensure(size_t count) {
    if (count <= n && p) return p;
    reset();
    check(cudaMalloc(&p, sizeof(T) * std::max<size_t>(count, 1)), "cudaMalloc");
    n = std::max<size_t>(count, 1);
    return p;
  }
};

// A resident mesh of instanced geometry.
struct DMeshRef {
  const float* pos;
  const float* nrm;      // or nullptr: face normals
  const float* uv;       // or nullptr: zeros
  const uint32_t* idx;   // or nullptr: not indexed
  int tri_count;
};

// An instance on the device: its world matrix, normal matrix (filled by
// k_instance_matrices) and per-triangle words.
struct DInstance {
  double world[16];
  double nm[9];
  int mesh, mirror, flags, side, flat;
  uint32_t material;
};

__device__ __forceinline__ void atomic_min_d(double* a, double v) {
  long long b = __double_as_longlong(v);
  if (b >= 0) {
    atomicMin(reinterpret_cast<long long*>(a), b);
  } else {
    atomicMax(reinterpret_cast<unsigned long long*>(a), static_cast<unsigned long long>(b));
  }
}
__device__ __forceinline__ void atomic_max_d(double* a, double v) {
  long long b = __double_as_longlong(v);
  if (b >= 0) {
    atomicMax(reinterpret_cast<long long*>(a), b);
  } else {
    atomicMin(reinterpret_cast<unsigned long long*>(a), static_cast<unsigned long long>(b));
  }
}

__host__ __device__ inline double area(double x0, double y0, double z0, double x1, double y1, double z1) {
  const double dx = x1 - x0, dy = y1 - y0, dz = z1 - z0;  // bvh.ts:180-183
  return dx * dy + dy * dz + dz * dx;
}

// Math.hypot as V8 computes it: scaled by the largest magnitude, summed with
// Kahan compensation.
__host__ __device__ inline double js_hypot3(double a, double b, double c) {
  const double x[3] = {fabs(a), fabs(b), fabs(c)};
  double mx = 0;
  for (int i = 0; i < 3; i++) {
    if (isinf(x[i])) return INFINITY;
  }
  for (int i = 0; i < 3; i++) {
    if (isnan(x[i])) return NAN;
    if (x[i] > mx) mx = x[i];
  }
  if (mx == 0) return 0;
  double sum = 0, comp = 0;
  for (int i = 0; i < 3; i++) {
    const double n = x[i] / mx;
    const double summand = n * n - comp;
    const double prelim = sum + summand;
    comp = (prelim - sum) - summand;
    sum = prelim;
  }
  return sqrt(sum) * mx;
}

// ------------------------------------------------------------------ build
// Two phases. Nodes of more than kSub triangles are split level by level,
// each level by two launches over segments of the level's triangles: k_bin
// bins a segment (several blocks of one node through exact atomics), and the
// last block of a node takes the split and queues the children; k_part moves
// the segment's triangles to their sides and gathers the children's bounds on
// the way. Counts, queues and offsets stay on the device, so the host only
// enqueues launches. Nodes of at most kSub triangles are then finished, all
// the way down, by one warp each in shared memory (k_subtrees).
//
// Triangles travel as what the build reads of them (box, centroid, index: 40
// bytes) instead of through an index array, so every pass streams.
//
// Numbering. The reference layout here is breadth first: the k-th inner node
// in (depth, first) order has its children at 1 + 2k and 2 + 2k. Nodes are
// found in no such order, so each inner node sets a bit at [depth][first], and
// a prefix count over the bits gives every k (k_rank_*, k_emit).
//
// Leaves tile the triangles, and the boundary before each leaf but the first
// is the split of exactly one inner node: both kinds of node are kept at such
// a position until they are numbered.
constexpr int kSub = 256;          // triangles of a subtree that one warp finishes
constexpr int kSubWarps = 2;       // warps of a block that finishes subtrees
constexpr int kSubTodo = 8;       // nodes of one that wait: each at least as large as all that came after it
constexpr int kSegMax = 4096;      // most triangles of a level kernel's segment (a multiple of kBuildBlock)
constexpr int kSegMin = 512;
constexpr unsigned kRootTag = 0xffffffffu;
constexpr int kLevels = kBuildDepth + 1;
constexpr int kRankGroup = 8;      // bitmap words per stored prefix

// Floats ordered as integers (min and max by integer atomics and reductions).
__device__ __forceinline__ int ordered(float f) {
  const int i = __float_as_int(f);
  return i ^ ((i >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float unordered(int i) { return __int_as_float(i ^ ((i >> 31) & 0x7fffffff)); }

// A triangle on its way through the build.
struct Prims {
  float4* a;  // box min xyz, box max x
  float4* b;  // box max yz, centroid xy
  float2* c;  // centroid z, triangle index
};

// A node of the level phase. box: node min xyz, max xyz, centroid min xyz,
// max xyz, as ordered integers. tag: twice the parent's first triangle, plus 1
// for a right child.
struct Node {
  int first, count, depth;
  unsigned tag;
  int seg0, nseg, acc;
  unsigned done;
  int box[12];
  int mode, axis, bin, nleft;  // the split: 0 binned, 1 the run in half
  double lo, scale;
  int child[2];  // index in the next level, or -1: a subtree
};

struct Subtree {
  int first, count, depth;
  unsigned tag;
  int parity;  // which buffer holds its triangles
};

// Bins of a node that several blocks share.
struct Acc {
  int cnt[3][kMaxBins];
  int bb[3][kMaxBins][6];
};

struct LevelCtl {
  int nodes, segs, accs;
};

struct BuildCtl {
  LevelCtl level[kLevels + 1];
  int subtrees, next_subtree;
  int inner_depth;   // deepest inner node, -1 for none
  // The depth that the reported level count goes by: of the deepest node that
  // is split, or is a leaf only by its cost, or is a small child of a node of
  // kWideMin triangles. The build itself does not use it.
  int slot_depth;
  int inner_nodes;   // set by k_rank_write
};

struct BuildState {
  BuildCtl* ctl;
  Prims prims[2];
  Node* nodes[2];
  int* segs[2];        // node of each segment
  int* seg_left;       // triangles going left in the node's segments before this one
  int* seg_cum;        // [segment][axis][bin]: triangles in bins <= bin
  Acc* acc[2];
  Subtree* subtrees;
  // Nodes by position, until they are numbered.
  float4 *inner_a, *inner_b, *leaf_a, *leaf_b;  // box min xyz, max x | max yz, first or count, depth (| axis << 8)
  unsigned *inner_t, *leaf_t;                   // tags
  unsigned* leaf_bits;                          // leaf starts
  unsigned* depth_bits;                         // [depth][first]: inner nodes
  int* rank;                                    // inner nodes before each group of kRankGroup words
  uint32_t* order;
  int n, words, seg, bins;                      // words: 32-bit words of one bitmap row
};

__device__ __forceinline__ void set_bit(unsigned* bits, size_t i) { atomicOr(bits + (i >> 5), 1u << (i & 31)); }

__device__ __forceinline__ void put_inner(const BuildState& st, int mid, const float* box, int first, int depth,
                                          int axis, unsigned tag) {
  st.inner_a[mid] = make_float4(box[0], box[1], box[2], box[3]);
  st.inner_b[mid] = make_float4(box[4], box[5], __int_as_float(first), __int_as_float(depth | (axis << 8)));
  st.inner_t[mid] = tag;
  set_bit(st.depth_bits, static_cast<size_t>(depth) * st.words * 32 + first);
}

__device__ __forceinline__ void put_leaf(const BuildState& st, int first, const float* box, int count, int depth,
                                         unsigned tag) {
  st.leaf_a[first] = make_float4(box[0], box[1], box[2], box[3]);
  st.leaf_b[first] = make_float4(box[4], box[5], __int_as_float(count), __int_as_float(depth));
  st.leaf_t[first] = tag;
}

__device__ __forceinline__ void add_prim(float* m, float4 a, float4 b, float cz) {
  m[0] = fminf(m[0], a.x); m[1] = fminf(m[1], a.y); m[2] = fminf(m[2], a.z);
  m[3] = fmaxf(m[3], a.w); m[4] = fmaxf(m[4], b.x); m[5] = fmaxf(m[5], b.y);
  m[6] = fminf(m[6], b.z); m[7] = fminf(m[7], b.w); m[8] = fminf(m[8], cz);
  m[9] = fmaxf(m[9], b.z); m[10] = fmaxf(m[10], b.w); m[11] = fmaxf(m[11], cz);
}

__device__ __forceinline__ bool is_max(int i) { return (i >= 3 && i < 6) || i >= 9; }

__device__ __forceinline__ void clear_box(float* m) {
#pragma unroll
  for (int i = 0; i < 12; i++) m[i] = is_max(i) ? -INFINITY : INFINITY;
}

// A box's bounds over the warp (every lane gets them), as ordered integers.
__device__ __forceinline__ int warp_bound(float v, bool max) {
  const int o = ordered(v);
  return max ? __reduce_max_sync(0xffffffffu, o) : __reduce_min_sync(0xffffffffu, o);
}

// A triangle's box and centroid (bvh.ts:22-33) into place i, and into the
// thread's bounds. A bound that is NaN (a vertex that is) is left out of every
// union, as the reference's comparisons leave it out: it is kept as the value
// that changes none, since min and max over ordered integers would take a NaN
// for the largest, and each split that keeps it would be lost. The centroid
// stays NaN and goes to the last bin.
__device__ __forceinline__ void put_prim(const Prims& p, int i, const float* o, float* m) {
  double lo[3], hi[3];
  for (int a = 0; a < 3; a++) {
    const double v0 = o[a], v1 = v0 + static_cast<double>(o[3 + a]), v2 = v0 + static_cast<double>(o[6 + a]);
    lo[a] = fmin(v0, fmin(v1, v2));
    hi[a] = fmax(v0, fmax(v1, v2));
  }
  const float4 a4 = make_float4(fminf(static_cast<float>(lo[0]), INFINITY), fminf(static_cast<float>(lo[1]), INFINITY),
                                fminf(static_cast<float>(lo[2]), INFINITY), fmaxf(static_cast<float>(hi[0]), -INFINITY));
  const float4 b4 = make_float4(fmaxf(static_cast<float>(hi[1]), -INFINITY), fmaxf(static_cast<float>(hi[2]), -INFINITY),
                                static_cast<float>((lo[0] + hi[0]) * 0.5), static_cast<float>((lo[1] + hi[1]) * 0.5));
  const float cz = static_cast<float>((lo[2] + hi[2]) * 0.5);
  p.a[i] = a4;
  p.b[i] = b4;
  p.c[i] = make_float2(cz, __int_as_float(i));
  add_prim(m, a4, b4, cz);
}

// The block's bounds into the root's.
__device__ __forceinline__ void put_root_bounds(const BuildState& st, const float* m) {
  __shared__ int red[12];
  if (threadIdx.x < 12) red[threadIdx.x] = ordered(is_max(threadIdx.x) ? -INFINITY : INFINITY);
  __syncthreads();
  for (int i = 0; i < 12; i++) {
    const int v = warp_bound(m[i], is_max(i));
    if ((threadIdx.x & 31) == 0) {
      if (is_max(i)) {
        atomicMax(&red[i], v);
      } else {
        atomicMin(&red[i], v);
      }
    }
  }
  __syncthreads();
  if (threadIdx.x < 12 && st.ctl->level[0].nodes > 0) {
    int* box = st.nodes[0][0].box;
    if (is_max(threadIdx.x)) {
      atomicMax(box + threadIdx.x, red[threadIdx.x]);
    } else {
      atomicMin(box + threadIdx.x, red[threadIdx.x]);
    }
  }
}

// Every triangle of `tris` (v0, e1, e2) into the build, and the root's bounds.
__global__ void __launch_bounds__(kBuildBlock) k_prepare(const float* __restrict__ tris, BuildState st) {
  float m[12];
  clear_box(m);
  for (int i = blockIdx.x * kBuildBlock + threadIdx.x; i < st.n; i += gridDim.x * kBuildBlock)
    put_prim(st.prims[0], i, tris + 9 * static_cast<size_t>(i), m);
  put_root_bounds(st, m);
}

// Math.min(bins - 1, Math.floor((c - lo) * scale)), bvh.ts:98: the product is
// never negative, so truncation is the floor; a NaN goes to the last bin.
__device__ __forceinline__ int bin_of(float c, double lo, double scale, int bins) {
  const double v = (static_cast<double>(c) - lo) * scale;
  return v < static_cast<double>(bins - 1) ? static_cast<int>(v) : bins - 1;
}

// Queues a node of the next level (the whole block; the node's index is the
// same in every thread).
__device__ void start_node(const BuildState& st, int level, int j, int first, int count, int depth, unsigned tag,
                           int seg0, int nseg, int acc) {
  Node& d = st.nodes[level & 1][j];
  const int tid = threadIdx.x;
  if (tid == 0) {
    d.first = first;
    d.count = count;
    d.depth = depth;
    d.tag = tag;
    d.seg0 = seg0;
    d.nseg = nseg;
    d.acc = acc;
    d.done = 0;
  }
  if (tid < 12) d.box[tid] = ordered(is_max(tid) ? -INFINITY : INFINITY);
  for (int i = tid; i < nseg; i += blockDim.x) st.segs[level & 1][seg0 + i] = j;
  if (acc >= 0) {
    Acc& a = st.acc[level & 1][acc];
    for (int i = tid; i < 3 * kMaxBins; i += blockDim.x) {
      (&a.cnt[0][0])[i] = 0;
      for (int q = 0; q < 6; q++) (&a.bb[0][0][0])[6 * i + q] = ordered(q < 3 ? INFINITY : -INFINITY);
    }
  }
}

// The root: a node of level 0, or a subtree of its own. One block; the
// control block is zeroed before it.
__global__ void __launch_bounds__(kBuildBlock) k_root(BuildState st) {
  if (st.n <= kSub) {
    if (threadIdx.x == 0) {
      st.subtrees[0] = Subtree{0, st.n, 0, kRootTag, 0};
      st.ctl->subtrees = 1;
    }
  } else {
    const int nseg = (st.n + st.seg - 1) / st.seg;
    if (threadIdx.x == 0) st.ctl->level[0] = LevelCtl{1, nseg, 1};
    start_node(st, 0, 0, 0, st.n, 0, kRootTag, 0, nseg, nseg > 1 ? 0 : -1);
  }
  if (threadIdx.x == 0) st.ctl->inner_depth = -1;
}

// A bin: its box as ordered integers, and its count. Seven words apart, the
// rows of 32 bins lie in different banks word by word (six apart, in pairs).
using BinRow = int[7];

__device__ __forceinline__ int empty_bin_word(int word) {
  return word == 6 ? 0 : ordered(word < 3 ? INFINITY : -INFINITY);
}

// Unions of a node's bins from the left (0) and from the right (1), per axis:
// [side][axis][k] covers bins [0, k] or [k, bins). Box bounds and counts, the
// boxes as ordered integers.
template <int MB>
struct Sweeps {
  int cnt[2][3][MB];
  int box[2][3][MB][6];
};

// The cheapest split of a node: after bin `split` of `axis`; axis < 0: no
// candidate.
struct Choice {
  double cost;
  int axis, split, nleft;
};

__device__ __forceinline__ double box_area(const int* b) {
  return area(unordered(b[0]), unordered(b[1]), unordered(b[2]), unordered(b[3]), unordered(b[4]), unordered(b[5]));
}

// The first minimum in (axis, split) order of the warp's candidates, each lane
// offering one (cost INFINITY: none), the same in every lane. Costs are ordered
// by their bits, flipped so that they compare as unsigned integers do (a set
// whose box is empty on one axis, its vertices being NaN there, has a cost of
// -INFINITY): three integer reductions instead of five rounds of double shuffles.
__device__ __forceinline__ Choice first_minimum(double cost, int axis, int split, int nleft) {
  const unsigned full = 0xffffffffu, sign = 0x80000000u;
  const unsigned flip = static_cast<unsigned>(__double2hiint(cost) >> 31);
  const unsigned hi = static_cast<unsigned>(__double2hiint(cost)) ^ (flip | sign);
  const unsigned lo = static_cast<unsigned>(__double2loint(cost)) ^ flip;
  const unsigned h = __reduce_min_sync(full, hi);
  const unsigned l = __reduce_min_sync(full, hi == h ? lo : ~0u);
  const unsigned at = __reduce_min_sync(full, hi == h && lo == l ? static_cast<unsigned>((axis << 8) | split) : ~0u);
  const unsigned back = h & sign ? 0u : ~0u;
  const double best = __hiloint2double(static_cast<int>(h ^ (back | sign)), static_cast<int>(l ^ back));
  if (!(best < INFINITY)) return Choice{INFINITY, -1, -1, 0};
  const unsigned who = __ballot_sync(full, hi == h && lo == l && static_cast<unsigned>((axis << 8) | split) == at);
  return Choice{best, static_cast<int>(at >> 8), static_cast<int>(at & 0xff), __shfl_sync(full, nleft, __ffs(who) - 1)};
}

// The cheapest split of a node's bins (bvh.ts:110-134), on one warp. Six lane
// groups sweep the three axes from both sides at once, a lane per pair of box
// bounds (and one for the counts), into shared memory; then each lane costs
// the splits after its bins. Min, max and sums are exact in any order and the
// areas and costs are the same expressions in double, so every candidate cost
// is the one-thread sweep's, and the first minimum wins, as there. Scans by
// shuffles of all seven values took three times the instructions.
template <int MB>
__device__ Choice best_split(const BinRow (*row)[MB], Sweeps<MB>& w, const bool* live, int bins) {
  const int lane = threadIdx.x & 31;
  if (lane < 24) {
    const int side = lane >= 12 ? 1 : 0, a = (lane - 12 * side) >> 2, q = lane & 3;
    int k = side ? bins - 1 : 0;
    const int step = side ? -1 : 1;
    if (q < 3) {
      int lo = ordered(INFINITY), hi = ordered(-INFINITY);
#pragma unroll 4
      for (int i = 0; i < bins; i++, k += step) {
        lo = min(lo, row[a][k][q]);
        hi = max(hi, row[a][k][3 + q]);
        w.box[side][a][k][q] = lo;
        w.box[side][a][k][3 + q] = hi;
      }
    } else {
      int c = 0;
#pragma unroll 4
      for (int i = 0; i < bins; i++, k += step) {
        c += row[a][k][6];
        w.cnt[side][a][k] = c;
      }
    }
  }
  __syncwarp();
  double best = INFINITY;
  int axis = 0, split = 0, nleft = 0;
  for (int c = lane; c < 3 * bins; c += 32) {
    const int a = c >= 2 * bins ? 2 : (c >= bins ? 1 : 0), k = c - a * bins;
    if (k >= bins - 1 || !live[a]) continue;
    const int lc = w.cnt[0][a][k], rc = w.cnt[1][a][k + 1];
    if (lc == 0 || rc == 0) continue;
    const double cost = lc * box_area(w.box[0][a][k]) + rc * box_area(w.box[1][a][k + 1]);
    if (cost < best) {  // false for a NaN
      best = cost;
      axis = a;
      split = k;
      nleft = lc;
    }
  }
  return first_minimum(best, axis, split, nleft);
}

// The choice (bvh.ts:137-163): mode -1 a SAH leaf, 0 the binned split, 1 the
// run in half (no candidate, or the bins put everything on one side).
__device__ __forceinline__ int choose(const Choice& c, const float* box, int count, int& axis, int& nleft) {
  axis = max(c.axis, 0);
  nleft = count >> 1;
  if (c.axis < 0) return 1;
  const double parent_area = area(box[0], box[1], box[2], box[3], box[4], box[5]);
  const double split_cost = 1 + (1 * c.cost) / fmax(parent_area, 1e-30);
  if (split_cost >= 1.0 * count && count <= 16) return -1;
  if (c.nleft == 0 || c.nleft == count) return 1;
  nleft = c.nleft;
  return 0;
}

__device__ __forceinline__ void binning(const float* cmin, const float* cmax, int bins, double* lo, double* scale,
                                        bool* live) {
  for (int a = 0; a < 3; a++) {
    lo[a] = cmin[a];
    const double extent = static_cast<double>(cmax[a]) - lo[a];
    live[a] = extent > 0;
    scale[a] = live[a] ? bins / extent : 0.0;
  }
}

__device__ __forceinline__ void bin_prim(int* row, const int* v) {
  atomicAdd(row + 6, 1);
  atomicMin(row, v[0]); atomicMin(row + 1, v[1]); atomicMin(row + 2, v[2]);
  atomicMax(row + 3, v[3]); atomicMax(row + 4, v[4]); atomicMax(row + 5, v[5]);
}

// The same where a bin takes many triangles: a bound is read first, without
// conflicts, and added to only if it grows. A bound read too early is smaller
// than it is by now, which costs an addition and changes nothing. (Not for a
// subtree's bins, of eight triangles at most on average: 16.4 M triangles
// rebuilt and traced 34.0 ms without, 34.6 with.)
__device__ __forceinline__ void bin_prim_checked(int* row, const int* v) {
  atomicAdd(row + 6, 1);
  const volatile int* now = row;
  int r[6];
  for (int q = 0; q < 6; q++) r[q] = now[q];
  for (int q = 0; q < 3; q++) {
    if (v[q] < r[q]) atomicMin(row + q, v[q]);
    if (v[3 + q] > r[3 + q]) atomicMax(row + 3 + q, v[3 + q]);
  }
}

// One segment of a level (see above). What bounds it: the latency of a node's
// steps at the lower levels, of loads and shared memory at the upper ones (0.21
// ms a level for 16.4 M triangles; reading them takes 0.09). A warp whose
// triangles all fall into one bin of an axis (neighbours in the model, at the
// upper levels) reduces them first and adds once; elsewhere a triangle adds to
// the bounds that it grows, few of a segment's (bin_prim_checked); the next
// triangle is loaded while one is binned. Adding to all six bounds of each bin,
// in rows of six words, was bound by the additions' conflicts: all levels
// together 7.4 -> 4.95 ms. 64 registers: 16.4 M triangles rebuilt and traced
// 40.1 ms, with 85 registers 40.7, with 128 41.3.
// B: 64 or 128 threads once a level has segments for every SM many times over
// (run_build): most of a small node's time is one warp's, the split's, and more
// and smaller blocks keep more nodes under way.
template <int B>
__global__ void __launch_bounds__(B, 1024 / B) k_bin(int level, BuildState st) {
  using Scan = cub::BlockScan<int, B>;
  __shared__ typename Scan::TempStorage scan_tmp;
  __shared__ BinRow row[3][kMaxBins];
  __shared__ Sweeps<kMaxBins> sweeps;
  __shared__ int s_flag, s_child[2], s_seg0[2], s_acc[2], s_mode, s_axis, s_bin, s_nleft;
  const unsigned full = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31;
  const int bins = st.bins, total = st.ctl->level[level].segs;
  const Prims p = st.prims[level & 1];
  for (int s = blockIdx.x; s < total; s += gridDim.x) {
    __syncthreads();  // the last segment's shared values are no longer read
    const int j = st.segs[level & 1][s];
    Node& nd = st.nodes[level & 1][j];
    const int nfirst = nd.first, ncount = nd.count, nseg = nd.nseg, seg = s - nd.seg0, depth = nd.depth;
    for (int i = tid; i < 3 * kMaxBins * 7; i += B) (&row[0][0][0])[i] = empty_bin_word(i % 7);
    double lo[3], scale[3];
    bool live[3];
    {
      float cmin[3], cmax[3];
      for (int i = 0; i < 3; i++) {
        cmin[i] = unordered(nd.box[6 + i]);
        cmax[i] = unordered(nd.box[9 + i]);
      }
      binning(cmin, cmax, bins, lo, scale, live);
    }
    __syncthreads();
    const int first = nfirst + seg * st.seg, end = min(nfirst + ncount, first + st.seg);
    float4 na = make_float4(INFINITY, INFINITY, INFINITY, -INFINITY);
    float4 nb = make_float4(-INFINITY, -INFINITY, 0.0f, 0.0f);
    float nc = 0.0f;
    const int got = first + tid;
    if (got < end) {
      na = p.a[got];
      nb = p.b[got];
      nc = p.c[got].x;
    }
    for (int base = first; base < end; base += B) {
      const int k = base + tid, ahead = k + B;
      const bool valid = k < end;
      const float4 a4 = valid ? na : make_float4(INFINITY, INFINITY, INFINITY, -INFINITY);
      const float4 b4 = valid ? nb : make_float4(-INFINITY, -INFINITY, 0.0f, 0.0f);
      const float cz = nc;
      if (ahead < end) {  // the next triangle is on its way while this one is binned
        na = p.a[ahead];
        nb = p.b[ahead];
        nc = p.c[ahead].x;
      }
      const int v[6] = {ordered(a4.x), ordered(a4.y), ordered(a4.z), ordered(a4.w), ordered(b4.x), ordered(b4.y)};
      const float c3[3] = {b4.z, b4.w, cz};
      const int here = __popc(__ballot_sync(full, valid));
      if (here == 0) continue;
      int w[6];
      bool reduced = false;
      for (int a = 0; a < 3; a++) {
        if (!live[a]) continue;
        const int b = valid ? bin_of(c3[a], lo[a], scale[a], bins) : 0;
        const int b0 = __shfl_sync(full, b, 0);  // lane 0 is valid when any is
        if (__all_sync(full, !valid || b == b0)) {
          if (!reduced) {
            for (int q = 0; q < 6; q++)
              w[q] = q < 3 ? __reduce_min_sync(full, v[q]) : __reduce_max_sync(full, v[q]);
            reduced = true;
          }
          if (lane == 0) {
            bin_prim(row[a][b0], w);
            if (here > 1) atomicAdd(&row[a][b0][6], here - 1);
          }
        } else if (valid) {
          bin_prim_checked(row[a][b], v);
        }
      }
    }
    __syncthreads();
    if (nseg > 1) {
      // This segment's cumulative counts, and its bins folded into the node's.
      Acc& acc = st.acc[level & 1][nd.acc];
      for (int a = tid >> 5; a < 3; a += B / 32) {
        int c = row[a][lane][6];
        for (int off = 1; off < 32; off <<= 1) {
          const int o = __shfl_up_sync(full, c, off);
          if (lane >= off) c += o;
        }
        st.seg_cum[(static_cast<size_t>(s) * 3 + a) * kMaxBins + lane] = c;
      }
      for (int i = tid; i < 3 * bins; i += B) {
        const int a = i / bins, b = i - a * bins;
        if (!live[a] || row[a][b][6] == 0) continue;
        atomicAdd(&acc.cnt[a][b], row[a][b][6]);
        for (int q = 0; q < 3; q++) {
          atomicMin(&acc.bb[a][b][q], row[a][b][q]);
          atomicMax(&acc.bb[a][b][3 + q], row[a][b][3 + q]);
        }
      }
      __threadfence();
      __syncthreads();
      if (tid == 0) s_flag = atomicAdd(&nd.done, 1u) == static_cast<unsigned>(nseg - 1) ? 1 : 0;
      __syncthreads();
      if (!s_flag) continue;
      __threadfence();
      for (int i = tid; i < 3 * kMaxBins; i += B) {
        (&row[0][0])[i][6] = __ldcg(&acc.cnt[0][0] + i);
        for (int q = 0; q < 6; q++) (&row[0][0])[i][q] = __ldcg(&acc.bb[0][0][0] + 6 * i + q);
      }
      __syncthreads();
    }
    if (tid < 32) {
      const Choice c = best_split<kMaxBins>(row, sweeps, live, bins);
      if (lane == 0) {
        float box[6];
        for (int i = 0; i < 6; i++) box[i] = unordered(nd.box[i]);
        int axis, nleft;
        const int mode = choose(c, box, ncount, axis, nleft);  // never a leaf: more than kSub triangles
        nd.mode = s_mode = mode;
        nd.axis = s_axis = axis;
        nd.bin = s_bin = c.split;
        nd.nleft = s_nleft = nleft;
        nd.lo = lo[axis];
        nd.scale = scale[axis];
        put_inner(st, nfirst + nleft, box, nfirst, depth, axis, nd.tag);
        atomicMax(&st.ctl->inner_depth, depth);
        const int kids[2] = {nleft, ncount - nleft};
        const bool last = depth + 1 >= kBuildDepth;
        int deepest = depth;
        for (int q = 0; q < 2; q++) {
          s_child[q] = -1;
          s_acc[q] = -1;
          if (kids[q] > kSub && !last) {
            const int ns = (kids[q] + st.seg - 1) / st.seg;
            LevelCtl& next = st.ctl->level[level + 1];
            s_child[q] = atomicAdd(&next.nodes, 1);
            s_seg0[q] = atomicAdd(&next.segs, ns);
            if (ns > 1) s_acc[q] = atomicAdd(&next.accs, 1);
          } else {
            const int t = atomicAdd(&st.ctl->subtrees, 1);
            st.subtrees[t] = Subtree{nfirst + (q ? nleft : 0), kids[q], depth + 1,
                                     2u * static_cast<unsigned>(nfirst) + q, (level + 1) & 1};
            if (ncount >= kWideMin) deepest = depth + 1;
          }
          nd.child[q] = s_child[q];
        }
        atomicMax(&st.ctl->slot_depth, deepest);
      }
    }
    __syncthreads();
    for (int q = 0; q < 2; q++) {
      if (s_child[q] < 0) continue;
      const int kc = q ? ncount - s_nleft : s_nleft;
      start_node(st, level + 1, s_child[q], nfirst + (q ? s_nleft : 0), kc, depth + 1,
                 2u * static_cast<unsigned>(nfirst) + q, s_seg0[q], (kc + st.seg - 1) / st.seg, s_acc[q]);
    }
    // Triangles going left before each of the node's segments.
    const int seg0 = s - seg;
    int running = 0;
    for (int base = 0; base < nseg; base += B) {
      const int i = base + tid;
      int left = 0;
      if (i < nseg && nseg > 1) {
        left = s_mode == 0 ? __ldcg(&st.seg_cum[(static_cast<size_t>(seg0 + i) * 3 + s_axis) * kMaxBins + s_bin])
                           : max(0, min(s_nleft - i * st.seg, min(st.seg, ncount - i * st.seg)));
      }
      int pre = 0, sum = 0;
      Scan(scan_tmp).ExclusiveSum(left, pre, sum);
      if (i < nseg) st.seg_left[seg0 + i] = running + pre;
      running += sum;
      __syncthreads();
    }
  }
}

// The stable partition of one segment (bvh.ts:145-171): each warp takes an
// equal share of it (at most 32 rounds: kSegMax / B), counts its lefts, and moves its triangles to the places its
// predecessors leave. What bounds it: DRAM at 16.4 M triangles (0.27 ms a level
// for 40 bytes read and written each, 74 % of the measured copy rate), the
// latency of its loads at a fifth of that.
template <int B>
__global__ void __launch_bounds__(B) k_part(int level, BuildState st) {
  static_assert(kSegMax / B <= 32, "a warp's rounds are its lanes");
  constexpr int kWarps = B / 32;
  __shared__ int s_lefts[kWarps];
  __shared__ int s_box[2][12];
  const unsigned full = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int total = st.ctl->level[level].segs;
  const Prims p = st.prims[level & 1], o = st.prims[(level + 1) & 1];
  for (int s = blockIdx.x; s < total; s += gridDim.x) {
    __syncthreads();
    const Node& nd = st.nodes[level & 1][st.segs[level & 1][s]];
    const int nfirst = nd.first, seg = s - nd.seg0, nleft = nd.nleft, mode = nd.mode, axis = nd.axis, bin = nd.bin;
    const double lo = nd.lo, scale = nd.scale;
    const int child[2] = {nd.child[0], nd.child[1]};
    const int first = nfirst + seg * st.seg, end = min(nfirst + nd.count, first + st.seg);
    if (tid < 24) (&s_box[0][0])[tid] = ordered(is_max(tid % 12) ? -INFINITY : INFINITY);
    const int rounds = (end - first + B - 1) / B;  // an equal share for every warp
    const int from = first + warp * 32 * rounds;
    unsigned mine = 0;  // lane r: the warp's round r, lanes going left
    for (int r = 0; r < rounds; r++) {
      const int k = from + 32 * r + lane;
      bool f = false;
      if (k < end) {
        if (mode == 0) {
          const float c = axis == 2 ? p.c[k].x : (axis == 0 ? p.b[k].z : p.b[k].w);
          f = bin_of(c, lo, scale, st.bins) <= bin;
        } else {
          f = k - nfirst < nleft;
        }
      }
      const unsigned b = __ballot_sync(full, f);
      if (lane == r) mine = b;
    }
    const int lefts = __reduce_add_sync(full, static_cast<unsigned>(__popc(mine)));
    if (lane == 0) s_lefts[warp] = lefts;
    __syncthreads();
    int before = 0;
    for (int w = 0; w < warp; w++) before += s_lefts[w];
    int lpos = nfirst + st.seg_left[s] + before;
    int rpos = nfirst + nleft + (from - nfirst) - (st.seg_left[s] + before);
    float ml[12], mr[12];
    clear_box(ml);
    clear_box(mr);
    for (int r = 0; r < rounds; r++) {
      const int k = from + 32 * r + lane;
      const unsigned b = __shfl_sync(full, mine, r);
      if (k < end) {
        const float4 a4 = p.a[k], b4 = p.b[k];
        const float2 c2 = p.c[k];
        const int pre = __popc(b & ((1u << lane) - 1u));
        const bool f = (b >> lane) & 1u;
        const int dst = f ? lpos + pre : rpos + (lane - pre);
        o.a[dst] = a4;
        o.b[dst] = b4;
        o.c[dst] = c2;
        if (f) {
          add_prim(ml, a4, b4, c2.x);
        } else {
          add_prim(mr, a4, b4, c2.x);
        }
      }
      lpos += __popc(b);
      rpos += max(0, min(32, end - (from + 32 * r))) - __popc(b);
    }
    for (int q = 0; q < 2; q++) {
      if (child[q] < 0) continue;  // a subtree takes its own bounds
      for (int i = 0; i < 12; i++) {
        const int v = warp_bound(q ? mr[i] : ml[i], is_max(i));
        if (lane == 0) {
          if (is_max(i)) {
            atomicMax(&s_box[q][i], v);
          } else {
            atomicMin(&s_box[q][i], v);
          }
        }
      }
    }
    __syncthreads();
    if (tid < 24) {
      const int q = tid / 12, i = tid - 12 * q;
      if (child[q] >= 0) {
        int* box = st.nodes[(level + 1) & 1][child[q]].box;
        if (is_max(i)) {
          atomicMax(box + i, s_box[q][i]);
        } else {
          atomicMin(box + i, s_box[q][i]);
        }
      }
    }
  }
}

// ---- subtrees

// A node of a subtree, positions within it. up: depth | parent's first << 8 |
// right << 16 | root << 17.
struct SubNode {
  int first, count;
  unsigned up;
  float box[6];
};

// Shared memory of a warp that finishes a subtree, for at most MB bins.
template <int MB>
struct SubWarp {
  float4 a[kSub];         // the triangles: box min xyz, max x
  float4 b[kSub];         // box max yz, centroid xy
  float c[kSub];          // centroid z
  BinRow row[3][MB];
  Sweeps<MB> sweeps;
  SubNode todo[kSubTodo];          // nodes of more than kTinyMax triangles
  uint2 tiny[kSub / (kMaxLeaf + 1) + 1];  // smaller ones: first | count << 16, SubNode::up
  uint8_t ord[kSub], moved[kSub];  // the triangles' order; a partition under way
};

__device__ __forceinline__ unsigned sub_tag(const Subtree& t, unsigned up) {
  if (up >> 17) return t.tag;
  return 2u * static_cast<unsigned>(t.first + ((up >> 8) & 0xff)) + ((up >> 16) & 1u);
}

__device__ __forceinline__ float centroid_of(float4 b, float c, int axis) { return axis == 2 ? c : (axis == 0 ? b.z : b.w); }

// binning() from a warp's centroid bounds (ordered integers), each axis's
// division on a lane of its own.
__device__ __forceinline__ void warp_binning(const int* cmin, const int* cmax, int bins, double* lo, double* scale,
                                             bool* live) {
  const unsigned full = 0xffffffffu;
  const int a = threadIdx.x & 3;
  const float mn = unordered(a == 0 ? cmin[0] : (a == 1 ? cmin[1] : cmin[2]));
  const float mx = unordered(a == 0 ? cmax[0] : (a == 1 ? cmax[1] : cmax[2]));
  const double extent = static_cast<double>(mx) - static_cast<double>(mn);
  const double sc = extent > 0 ? bins / extent : 0.0;
  for (int q = 0; q < 3; q++) {
    lo[q] = unordered(cmin[q]);
    scale[q] = __shfl_sync(full, sc, q);
    live[q] = unordered(cmax[q]) > unordered(cmin[q]);  // the difference of two floats is never rounded to 0
  }
}

// A node of more than kTinyMax triangles: its bins, their sweeps and the
// partition. Returns the split's mode (-1: a SAH leaf) with axis and nleft; the
// children's boxes are sweeps.box[0][axis][left_at] and [1][axis][left_at + 1].
template <int MB>
__device__ int sub_split(const BuildState& st, SubWarp<MB>& w, const SubNode& e, int& axis, int& nleft, int& left_at) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int f = e.first, n = e.count, bins = st.bins;
  float cmn[3] = {INFINITY, INFINITY, INFINITY}, cmx[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (int k = lane; k < n; k += 32) {
    const int id = w.ord[f + k];
    const float4 b = w.b[id];
    const float c = w.c[id];
    cmn[0] = fminf(cmn[0], b.z); cmn[1] = fminf(cmn[1], b.w); cmn[2] = fminf(cmn[2], c);
    cmx[0] = fmaxf(cmx[0], b.z); cmx[1] = fmaxf(cmx[1], b.w); cmx[2] = fmaxf(cmx[2], c);
  }
  int cmin[3], cmax[3];
  for (int q = 0; q < 3; q++) {
    cmin[q] = __reduce_min_sync(full, ordered(cmn[q]));
    cmax[q] = __reduce_max_sync(full, ordered(cmx[q]));
  }
  double lo[3], scale[3];
  bool live[3];
  warp_binning(cmin, cmax, bins, lo, scale, live);
  for (int i = lane; i < 3 * MB; i += 32) {
    for (int q = 0; q < 7; q++) (&w.row[0][0])[i][q] = empty_bin_word(q);
  }
  __syncwarp();
  for (int k = lane; k < n; k += 32) {
    const int id = w.ord[f + k];
    const float4 a = w.a[id], b = w.b[id];
    const float c = w.c[id];
    const int v[6] = {ordered(a.x), ordered(a.y), ordered(a.z), ordered(a.w), ordered(b.x), ordered(b.y)};
    for (int q = 0; q < 3; q++) {
      if (!live[q]) continue;
      const int x = bin_of(centroid_of(b, c, q), lo[q], scale[q], bins);
      bin_prim(w.row[q][x], v);
    }
  }
  __syncwarp();
  const Choice c = best_split<MB>(w.row, w.sweeps, live, bins);
  const int mode = choose(c, e.box, n, axis, nleft);
  if (mode < 0) return mode;
  left_at = c.split;
  const double l = axis == 0 ? lo[0] : (axis == 1 ? lo[1] : lo[2]);
  const double sc = axis == 0 ? scale[0] : (axis == 1 ? scale[1] : scale[2]);
  int lpos = 0, rpos = nleft;
  for (int base = 0; base < n; base += 32) {
    const int k = base + lane;
    const bool valid = k < n;
    const int id = valid ? w.ord[f + k] : 0;
    const bool left = valid && (mode == 0 ? bin_of(centroid_of(w.b[id], w.c[id], axis), l, sc, bins) <= c.split : k < nleft);
    const unsigned b = __ballot_sync(full, left);
    const int pre = __popc(b & ((1u << lane) - 1u));
    if (valid) w.moved[left ? lpos + pre : rpos + (lane - pre)] = static_cast<uint8_t>(id);
    lpos += __popc(b);
    rpos += min(32, n - base) - __popc(b);
  }
  __syncwarp();
  for (int k = lane; k < n; k += 32) w.ord[f + k] = w.moved[k];
  __syncwarp();
  return mode;
}

// A box that one lane grows.
struct LaneBox {
  float b[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  __device__ __forceinline__ void add(float4 p, float4 q) {
    b[0] = fminf(b[0], p.x); b[1] = fminf(b[1], p.y); b[2] = fminf(b[2], p.z);
    b[3] = fmaxf(b[3], p.w); b[4] = fmaxf(b[4], q.x); b[5] = fmaxf(b[5], q.y);
  }
  __device__ __forceinline__ double size() const { return area(b[0], b[1], b[2], b[3], b[4], b[5]); }
};

// A node of at most kTinyMax triangles and everything below it, by one lane,
// while the other lanes do theirs: a warp per such node leaves three quarters
// of its lanes idle and pays every warp-wide step for a few triangles. No bins
// either: per axis the lane sorts the triangles by bin, and sweeps them from
// the right (areas kept) and from the left. At the last triangle of each
// occupied bin b these give the left set {bins <= b} and the right set
// {bins > b} of the split after b. Split positions between occupied bins have
// the same two sets and so the same cost as the occupied bin before them, and
// positions before the first or from the last occupied bin leave a side empty,
// so the first minimum over these candidates in (axis, split) order is the
// binned sweep's: the same costs from the same unions, the same choice.
// `inner_deep`, `slot_deep`: as in BuildCtl.
template <int MB>
__device__ void lane_subtree(const BuildState& st, const Subtree& t, SubWarp<MB>& w, uint2 root, int& inner_deep,
                             int& slot_deep) {
  int key[kTinyMax];         // bin << 8 | triangle, in bin order
  double right[kTinyMax];    // area of the triangles from here on
  uint2 wait[2];             // the larger child waits: at most log2(12 / 5) of them
  int waiting = 0;
  uint2 e = root;
  const int bins = st.bins;
  for (;;) {
    const int f = e.x & 0xff, n = e.x >> 16, depth = e.y & 0xff;
    LaneBox box;
    float cmn[3] = {INFINITY, INFINITY, INFINITY}, cmx[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int k = 0; k < n; k++) {
      const int id = w.ord[f + k];
      const float4 a = w.a[id], b = w.b[id];
      const float c = w.c[id];
      box.add(a, b);
      cmn[0] = fminf(cmn[0], b.z); cmn[1] = fminf(cmn[1], b.w); cmn[2] = fminf(cmn[2], c);
      cmx[0] = fmaxf(cmx[0], b.z); cmx[1] = fmaxf(cmx[1], b.w); cmx[2] = fmaxf(cmx[2], c);
    }
    Choice best{INFINITY, -1, 0, 0};
    double best_lo = 0, best_scale = 0;
#pragma unroll 1
    for (int q = 0; q < 3; q++) {
      const double lo = q == 0 ? cmn[0] : (q == 1 ? cmn[1] : cmn[2]);
      const double extent = static_cast<double>(q == 0 ? cmx[0] : (q == 1 ? cmx[1] : cmx[2])) - lo;
      if (!(extent > 0)) continue;
      const double scale = bins / extent;
      for (int k = 0; k < n; k++) {
        const int id = w.ord[f + k];
        const int b = bin_of(centroid_of(w.b[id], w.c[id], q), lo, scale, bins);
        int j = k;
        for (; j > 0 && (key[j - 1] >> 8) > b; j--) key[j] = key[j - 1];
        key[j] = (b << 8) | id;
      }
      LaneBox r;
      for (int k = n - 1; k > 0; k--) {
        const int id = key[k] & 0xff;
        r.add(w.a[id], w.b[id]);
        right[k] = r.size();
      }
      LaneBox l;
      int at = key[0];
      for (int k = 0; k < n - 1; k++) {
        const int id = at & 0xff, b = at >> 8;
        l.add(w.a[id], w.b[id]);
        at = key[k + 1];
        if (b == (at >> 8)) continue;
        const double cost = (k + 1) * l.size() + (n - k - 1) * right[k + 1];
        if (cost < best.cost) {  // false for a NaN
          best = Choice{cost, q, b, k + 1};
          best_lo = lo;
          best_scale = scale;
        }
      }
    }
    int axis, nleft;
    const int mode = choose(best, box.b, n, axis, nleft);
    bool next = false;
    if (mode < 0) {
      put_leaf(st, t.first + f, box.b, n, depth, sub_tag(t, e.y));
      set_bit(st.leaf_bits, t.first + f);
      slot_deep = max(slot_deep, depth);
    } else {
      put_inner(st, t.first + f + nleft, box.b, t.first + f, depth, axis, sub_tag(t, e.y));
      inner_deep = max(inner_deep, depth);
      // The stable partition, and the children's boxes if they are leaves.
      LaneBox kid[2];
      int lpos = 0, rpos = nleft;
      for (int k = 0; k < n; k++) key[k] = w.ord[f + k];
      for (int k = 0; k < n; k++) {
        const int id = key[k];
        const float4 b = w.b[id];
        const bool left = mode == 0 ? bin_of(centroid_of(b, w.c[id], axis), best_lo, best_scale, bins) <= best.split
                                    : k < nleft;
        if (left) {
          kid[0].add(w.a[id], b);
          w.ord[f + lpos++] = static_cast<uint8_t>(id);
        } else {
          kid[1].add(w.a[id], b);
          w.ord[f + rpos++] = static_cast<uint8_t>(id);
        }
      }
      const bool last = depth + 1 >= kBuildDepth;
      uint2 keep = make_uint2(0, 0);
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const int kf = f + (q ? nleft : 0), kc = q ? n - nleft : nleft;
        const unsigned up = static_cast<unsigned>(depth + 1) | (f << 8) | (q << 16);
        if (last || kc <= kMaxLeaf) {
          put_leaf(st, t.first + kf, kid[q].b, kc, depth + 1, sub_tag(t, up));
          set_bit(st.leaf_bits, t.first + kf);
        } else if (!next) {
          keep = make_uint2(kf | (kc << 16), up);
          next = true;
        } else {
          const uint2 other = make_uint2(kf | (kc << 16), up);
          const bool bigger = kc > static_cast<int>(keep.x >> 16);
          wait[waiting++] = bigger ? other : keep;
          keep = bigger ? keep : other;
        }
      }
      if (next) e = keep;
    }
    if (next) continue;
    if (waiting == 0) break;
    e = wait[--waiting];
  }
}

// The bounds of triangles [first, first + count) of the order, in every lane.
template <int MB>
__device__ void sub_bounds(SubWarp<MB>& w, int first, int count, float* box) {
  float m[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  for (int k = threadIdx.x & 31; k < count; k += 32) {
    const int id = w.ord[first + k];
    const float4 a = w.a[id], b = w.b[id];
    m[0] = fminf(m[0], a.x); m[1] = fminf(m[1], a.y); m[2] = fminf(m[2], a.z);
    m[3] = fmaxf(m[3], a.w); m[4] = fmaxf(m[4], b.x); m[5] = fmaxf(m[5], b.y);
  }
  for (int q = 0; q < 6; q++) box[q] = unordered(warp_bound(m[q], is_max(q)));
}

// Finishes subtrees, one warp each, from a queue: a depth-first walk over its
// larger nodes, the smaller child first (so few nodes wait), then a lane per
// tiny node, then the order of the triangles. What bounds it: issue slots and
// shared-memory latency, at the warps that shared memory leaves room for; only
// the triangles in and the nodes out touch DRAM.
template <int MB>
__global__ void __launch_bounds__(32 * kSubWarps) k_subtrees(BuildState st) {
  extern __shared__ __align__(16) unsigned char smem[];
  SubWarp<MB>& w = reinterpret_cast<SubWarp<MB>*>(smem)[threadIdx.x >> 5];
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int count = st.ctl->subtrees;
  int inner_deep = -1, slot_deep = 0;
  for (;;) {
    int s = 0;
    if (lane == 0) s = atomicAdd(&st.ctl->next_subtree, 1);
    s = __shfl_sync(full, s, 0);
    if (s >= count) break;
    const Subtree t = st.subtrees[s];
    const Prims p = st.prims[t.parity];
    const int n = t.count;
    if (n <= kMaxLeaf || t.depth >= kBuildDepth) {  // a leaf; at the depth limit of any size
      float m[12];
      clear_box(m);
      for (int k = lane; k < n; k += 32) {
        const float4 a4 = p.a[t.first + k], b4 = p.b[t.first + k];
        const float2 c2 = p.c[t.first + k];
        add_prim(m, a4, b4, c2.x);
        st.order[t.first + k] = __float_as_int(c2.y);
      }
      float box[6];
      for (int q = 0; q < 6; q++) box[q] = unordered(warp_bound(m[q], is_max(q)));
      if (lane == 0) {
        put_leaf(st, t.first, box, n, t.depth, t.tag);
        set_bit(st.leaf_bits, t.first);
      }
      continue;
    }
    __syncwarp();
    for (int k = lane; k < n; k += 32) {
      w.a[k] = p.a[t.first + k];
      w.b[k] = p.b[t.first + k];
      w.c[k] = p.c[t.first + k].x;
      w.ord[k] = static_cast<uint8_t>(k);
    }
    __syncwarp();
    SubNode e{0, n, static_cast<unsigned>(t.depth) | (1u << 17), {}};
    int waiting = 0, tiny = 0;
    bool next = n > kTinyMax;
    if (next) {
      sub_bounds(w, 0, n, e.box);
    } else {
      if (lane == 0) w.tiny[0] = make_uint2(n << 16, e.up);
      tiny = 1;
    }
    while (next) {
      const int depth = static_cast<int>(e.up & 0xff);
      int axis, nleft, left_at;
      const int mode = sub_split(st, w, e, axis, nleft, left_at);
      const bool last = depth + 1 >= kBuildDepth;
      SubNode keep{};
      next = false;
      if (mode < 0) {
        if (lane == 0) {
          put_leaf(st, t.first + e.first, e.box, e.count, depth, sub_tag(t, e.up));
          set_bit(st.leaf_bits, t.first + e.first);
        }
        slot_deep = max(slot_deep, depth);
      } else {
        if (lane == 0)
          put_inner(st, t.first + e.first + nleft, e.box, t.first + e.first, depth, axis, sub_tag(t, e.up));
        inner_deep = max(inner_deep, depth);
      }
#pragma unroll
      for (int q = 0; q < 2 && mode >= 0; q++) {
        SubNode kid{e.first + (q ? nleft : 0), q ? e.count - nleft : nleft,
                    static_cast<unsigned>(depth + 1) | (e.first << 8) | (q << 16), {}};
        const bool leaf = last || kid.count <= kMaxLeaf;
        if (!leaf && kid.count <= kTinyMax) {
          if (lane == 0) w.tiny[tiny] = make_uint2(kid.first | (kid.count << 16), kid.up);
          tiny++;
          continue;
        }
        if (mode == 0) {
          for (int i = 0; i < 6; i++) kid.box[i] = unordered(w.sweeps.box[q][axis][left_at + q][i]);
        } else {
          sub_bounds(w, kid.first, kid.count, kid.box);
        }
        if (leaf) {
          if (lane == 0) {
            put_leaf(st, t.first + kid.first, kid.box, kid.count, depth + 1, sub_tag(t, kid.up));
            set_bit(st.leaf_bits, t.first + kid.first);
          }
        } else if (!next) {
          keep = kid;
          next = true;
        } else {
          const bool bigger = kid.count > keep.count;
          if (lane == 0) w.todo[waiting] = bigger ? kid : keep;
          waiting++;
          if (!bigger) keep = kid;
        }
      }
      __syncwarp();  // the sweeps are read, the lists written
      if (next) {
        e = keep;
      } else if (waiting > 0) {
        e = w.todo[--waiting];
        next = true;
        __syncwarp();
      }
    }
    __syncwarp();
    for (int k = lane; k < tiny; k += 32) lane_subtree(st, t, w, w.tiny[k], inner_deep, slot_deep);
    __syncwarp();
    for (int k = lane; k < n; k += 32) st.order[t.first + k] = __float_as_int(p.c[t.first + w.ord[k]].y);
    __syncwarp();
  }
  inner_deep = __reduce_max_sync(full, inner_deep);
  slot_deep = __reduce_max_sync(full, slot_deep);
  if (lane == 0) {
    if (inner_deep >= 0) atomicMax(&st.ctl->inner_depth, inner_deep);
    atomicMax(&st.ctl->slot_depth, max(slot_deep, inner_deep));
  }
}

// ---- numbering
constexpr int kScanBlocks = 4 * 148;
constexpr int kScanThreads = 256;

__device__ __forceinline__ void scan_segment(long long n, long long& lo, long long& hi) {
  const long long seg = (n + kScanBlocks - 1) / kScanBlocks;
  lo = min(n, static_cast<long long>(blockIdx.x) * seg);
  hi = min(n, lo + seg);
}

__device__ __forceinline__ long long rank_groups(const BuildState& st) {
  return (static_cast<long long>(st.ctl->inner_depth + 1) * st.words + kRankGroup - 1) / kRankGroup;
}

__device__ __forceinline__ int group_bits(const unsigned* bits, long long g) {
  const uint4* w = reinterpret_cast<const uint4*>(bits + kRankGroup * g);
  const uint4 x = w[0], y = w[1];
  return __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w) + __popc(y.x) + __popc(y.y) + __popc(y.z) + __popc(y.w);
}

__global__ void __launch_bounds__(kScanThreads) k_rank_sums(BuildState st, int* __restrict__ sums) {
  using Reduce = cub::BlockReduce<int, kScanThreads>;
  __shared__ typename Reduce::TempStorage tmp;
  long long lo, hi;
  scan_segment(rank_groups(st), lo, hi);
  int v = 0;
  for (long long g = lo + threadIdx.x; g < hi; g += kScanThreads) v += group_bits(st.depth_bits, g);
  const int total = Reduce(tmp).Sum(v);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads) k_rank_write(BuildState st, const int* __restrict__ sums) {
  using Reduce = cub::BlockReduce<int, kScanThreads>;
  using Scan = cub::BlockScan<int, kScanThreads>;
  __shared__ union {
    typename Reduce::TempStorage reduce;
    typename Scan::TempStorage scan;
  } tmp;
  __shared__ int base;
  long long lo, hi;
  scan_segment(rank_groups(st), lo, hi);
  int before = 0;
  for (int b = static_cast<int>(threadIdx.x); b < static_cast<int>(blockIdx.x); b += kScanThreads) before += sums[b];
  const int offset = Reduce(tmp.reduce).Sum(before);
  if (threadIdx.x == 0) base = offset;
  __syncthreads();
  int running = base;
  if (blockIdx.x == kScanBlocks - 1 && threadIdx.x == 0) st.ctl->inner_nodes = running + sums[kScanBlocks - 1];
  for (long long tile = lo; tile < hi; tile += kScanThreads) {
    const long long g = tile + threadIdx.x;
    const int v = g < hi ? group_bits(st.depth_bits, g) : 0;
    int ex = 0, total = 0;
    Scan(tmp.scan).ExclusiveSum(v, ex, total);
    if (g < hi) st.rank[g] = running + ex;
    running += total;
    __syncthreads();
  }
}

// Inner nodes before the one at [depth][first], breadth first.
__device__ __forceinline__ int inner_rank(const BuildState& st, int depth, int first) {
  const long long word = static_cast<long long>(depth) * st.words + (first >> 5);
  const long long g = word / kRankGroup;
  int r = st.rank[g];
  for (long long q = g * kRankGroup; q < word; q++) r += __popc(st.depth_bits[q]);
  return r + __popc(st.depth_bits[word] & ((1u << (first & 31)) - 1u));
}

__device__ __forceinline__ int node_index(const BuildState& st, unsigned tag, int depth) {
  return tag == kRootTag ? 0 : 1 + 2 * inner_rank(st, depth - 1, static_cast<int>(tag >> 1)) + static_cast<int>(tag & 1u);
}

__device__ __forceinline__ void write_node(int i, float4 a, float4 b, int x, int y, int z, float* __restrict__ bounds,
                                           int* __restrict__ nodes) {
  float* bo = bounds + 6 * static_cast<size_t>(i);
  bo[0] = a.x; bo[1] = a.y; bo[2] = a.z;
  bo[3] = a.w; bo[4] = b.x; bo[5] = b.y;
  int* nd = nodes + 3 * static_cast<size_t>(i);
  nd[0] = x; nd[1] = y; nd[2] = z;
}

// The leaf that starts at each position, and the inner node that splits there.
__global__ void __launch_bounds__(256) k_emit(BuildState st, float* __restrict__ bounds, int* __restrict__ nodes) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= st.n || !((st.leaf_bits[k >> 5] >> (k & 31)) & 1u)) return;
  const float4 la = st.leaf_a[k], lb = st.leaf_b[k];
  write_node(node_index(st, st.leaf_t[k], __float_as_int(lb.w)), la, lb, k, __float_as_int(lb.z), 0, bounds, nodes);
  if (k == 0) return;
  const float4 a = st.inner_a[k], b = st.inner_b[k];
  const int first = __float_as_int(b.z), depth = __float_as_int(b.w) & 0xff, axis = __float_as_int(b.w) >> 8;
  write_node(node_index(st, st.inner_t[k], depth), a, b, 1 + 2 * inner_rank(st, depth, first), 0, axis, bounds, nodes);
}

// ---- compile (src/compile.ts:336-343 and 359-432)

// Float32 triangles from the sink's doubles, and the largest coordinate.
__global__ void k_sink_triangles(const double* __restrict__ p, int n, float* __restrict__ tris,
                                 unsigned long long* __restrict__ max_coord) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double mc = 0;
  if (i < n) {
    const double* q = p + 9 * static_cast<size_t>(i);
    float* t = tris + 9 * static_cast<size_t>(i);
    for (int a = 0; a < 3; a++) {
      t[a] = static_cast<float>(q[a]);
      t[3 + a] = static_cast<float>(q[3 + a] - q[a]);
      t[6 + a] = static_cast<float>(q[6 + a] - q[a]);
    }
    for (int k = 0; k < 9; k++) mc = fmax(mc, fabs(q[k]));
  }
  for (int off = 16; off > 0; off >>= 1) mc = fmax(mc, __shfl_xor_sync(0xffffffffu, mc, off));
  if ((threadIdx.x & 31) == 0) atomicMax(max_coord, static_cast<unsigned long long>(__double_as_longlong(mc)));
}

// Everything in BVH order (compile.ts:364-377).
__global__ void k_reorder(const uint32_t* __restrict__ order, int n, const float* __restrict__ tris_in,
                          const double* __restrict__ nrm, const double* __restrict__ uv,
                          const double* __restrict__ colors, const uint8_t* __restrict__ has_color, int any_colors,
                          const uint32_t* __restrict__ mats, const uint8_t* __restrict__ flags,
                          const uint8_t* __restrict__ sides, float* __restrict__ tris_out,
                          float* __restrict__ nrm_out, float* __restrict__ uv_out, float* __restrict__ col_out,
                          uint32_t* __restrict__ mats_out, uint8_t* __restrict__ flags_out,
                          uint8_t* __restrict__ sides_out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const size_t s = order[i];
  for (int k = 0; k < 9; k++) tris_out[9 * static_cast<size_t>(i) + k] = tris_in[9 * s + k];
  for (int k = 0; k < 9; k++) nrm_out[9 * static_cast<size_t>(i) + k] = static_cast<float>(nrm[9 * s + k]);
  for (int k = 0; k < 6; k++) uv_out[6 * static_cast<size_t>(i) + k] = static_cast<float>(uv[6 * s + k]);
  if (any_colors) {
    for (int k = 0; k < 12; k++)
      col_out[12 * static_cast<size_t>(i) + k] = has_color[s] ? static_cast<float>(colors[12 * s + k]) : 1.0f;
  }
  mats_out[i] = mats[s];
  flags_out[i] = flags[s];
  sides_out[i] = sides[s];
}

// The vertex bounding box of a grid's threads (compile.ts:378-385): each block
// reduces its own, then one atomic per bound.
struct VertexBox {
  double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  __device__ __forceinline__ void add(const float* o) {
    for (int v = 0; v < 3; v++) {
      for (int a = 0; a < 3; a++) {
        const double x = static_cast<double>(o[a]) + (v == 1 ? o[3 + a] : v == 2 ? o[6 + a] : 0.0f);
        lo[a] = fmin(lo[a], x);
        hi[a] = fmax(hi[a], x);
      }
    }
  }
  __device__ __forceinline__ void reduce(double* box) {
    __shared__ double red[kBuildBlock / 32][6];
    for (int off = 16; off > 0; off >>= 1) {
      for (int a = 0; a < 3; a++) {
        lo[a] = fmin(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], off));
        hi[a] = fmax(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], off));
      }
    }
    if ((threadIdx.x & 31) == 0) {
      for (int a = 0; a < 3; a++) {
        red[threadIdx.x >> 5][a] = lo[a];
        red[threadIdx.x >> 5][3 + a] = hi[a];
      }
    }
    __syncthreads();
    if (threadIdx.x < 6) {
      double v = red[0][threadIdx.x];
      for (int w = 1; w < kBuildBlock / 32; w++)
        v = threadIdx.x < 3 ? fmin(v, red[w][threadIdx.x]) : fmax(v, red[w][threadIdx.x]);
      if (threadIdx.x < 3) {
        atomic_min_d(box + threadIdx.x, v);
      } else {
        atomic_max_d(box + threadIdx.x, v);
      }
    }
  }
};

// writeTangent (compile.ts:406-432) of a triangle (v0, e1, e2) with its uvs.
__device__ float4 tangent_of(const float* o, const float* u6) {
  const double e1x = o[3], e1y = o[4], e1z = o[5], e2x = o[6], e2y = o[7], e2z = o[8];
  const double du1 = static_cast<double>(u6[2]) - u6[0], dv1 = static_cast<double>(u6[3]) - u6[1];
  const double du2 = static_cast<double>(u6[4]) - u6[0], dv2 = static_cast<double>(u6[5]) - u6[1];
  const double nx = e1y * e2z - e1z * e2y, ny = e1z * e2x - e1x * e2z, nz = e1x * e2y - e1y * e2x;
  const double d = du1 * dv2 - du2 * dv1;
  double tx, ty, tz, sign = 1;
  if (fabs(d) > 1e-20) {
    const double r = 1 / d;
    tx = (e1x * dv2 - e2x * dv1) * r;
    ty = (e1y * dv2 - e2y * dv1) * r;
    tz = (e1z * dv2 - e2z * dv1) * r;
    const double bx = (e2x * du1 - e1x * du2) * r, by = (e2y * du1 - e1y * du2) * r, bz = (e2z * du1 - e1z * du2) * r;
    const double cx = ny * tz - nz * ty, cy = nz * tx - nx * tz, cz = nx * ty - ny * tx;
    sign = cx * bx + cy * by + cz * bz < 0 ? -1 : 1;
  } else if (fabs(nx) < 0.9 * js_hypot3(nx, ny, nz)) {
    tx = 0; ty = -nz; tz = ny;
  } else {
    tx = nz; ty = 0; tz = -nx;
  }
  double length = js_hypot3(tx, ty, tz);
  if (length == 0 || isnan(length)) length = 1;
  return make_float4(static_cast<float>(tx / length), static_cast<float>(ty / length), static_cast<float>(tz / length),
                     static_cast<float>(sign));
}

__global__ void __launch_bounds__(kBuildBlock) k_tangents(const float* __restrict__ tris, const float* __restrict__ uvs,
                                                          int n, float4* __restrict__ tangents, double* __restrict__ box) {
  VertexBox vb;
  for (int i = blockIdx.x * kBuildBlock + threadIdx.x; i < n; i += gridDim.x * kBuildBlock) {
    const float* o = tris + 9 * static_cast<size_t>(i);
    vb.add(o);
    tangents[i] = tangent_of(o, uvs + 6 * static_cast<size_t>(i));
  }
  vb.reduce(box);
}

int blocks_of(long long n, int b) { return static_cast<int>((n + b - 1) / b); }

// ---- instanced geometry on the device (addMesh, src/compile.ts:212-306)

// normalMatrix, src/compile.ts:192-205: cofactors divided by the determinant,
// evaluated in the reference's order (this file is compiled without FMA).
__global__ void k_instance_matrices(DInstance* __restrict__ inst, int count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  DInstance& d = inst[i];
  const double* m = d.world;
  const double a = m[0], b = m[4], c = m[8], dd = m[1], e = m[5], f = m[9], g = m[2], h = m[6], ii = m[10];
  const double A = e * ii - f * h, B = -(dd * ii - f * g), C = dd * h - e * g;
  const double det = a * A + b * B + c * C;
  const double sc = det != 0 ? 1 / det : 0;
  d.nm[0] = A * sc; d.nm[1] = (-(b * ii - c * h)) * sc; d.nm[2] = (b * f - c * e) * sc;
  d.nm[3] = B * sc; d.nm[4] = (a * ii - c * g) * sc; d.nm[5] = (-(a * f - c * dd)) * sc;
  d.nm[6] = C * sc; d.nm[7] = (-(a * h - b * g)) * sc; d.nm[8] = (a * e - b * dd) * sc;
  d.mirror = det < 0 ? 1 : 0;
}

// Instances and meshes as the kernels below see them; base: the first
// triangle of each instance, then the total.
struct Instances {
  const DInstance* inst;
  const DMeshRef* meshes;
  const int* base;
  int count;
};

// Triangle i's instance: the last one that starts at or before it and is not
// empty.
__device__ __forceinline__ int instance_of(const Instances& in, int i) {
  int lo = 0, hi = in.count - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (in.base[mid] <= i) {
      lo = mid;
    } else {
      hi = mid - 1;
    }
  }
  return lo;
}

// World-space vertices of triangle k of an instance in double (addMesh,
// compile.ts:212-306), its vertex indices, and float32 v0 / e1 / e2 as the
// compile's Float32Array stores make them (compile.ts:337-343).
__device__ __forceinline__ void world_triangle(const DInstance& d, const DMeshRef& mr, int k, int* ids, double* p,
                                               float* t) {
  for (int v = 0; v < 3; v++) ids[v] = 3 * k + v;
  if (mr.idx) {
    for (int v = 0; v < 3; v++) ids[v] = static_cast<int>(mr.idx[ids[v]]);
  }
  if (d.mirror) {  // a mirroring transform reverses the winding
    const int x = ids[1];
    ids[1] = ids[2];
    ids[2] = x;
  }
  const double* w = d.world;
  for (int v = 0; v < 3; v++) {
    const float* q = mr.pos + 3 * static_cast<size_t>(ids[v]);
    const double x = q[0], y = q[1], z = q[2];
    p[3 * v] = w[0] * x + w[4] * y + w[8] * z + w[12];
    p[3 * v + 1] = w[1] * x + w[5] * y + w[9] * z + w[13];
    p[3 * v + 2] = w[2] * x + w[6] * y + w[10] * z + w[14];
  }
  for (int a = 0; a < 3; a++) {
    t[a] = static_cast<float>(p[a]);
    t[3 + a] = static_cast<float>(p[3 + a] - p[a]);
    t[6 + a] = static_cast<float>(p[6 + a] - p[a]);
  }
}

// Every instance's triangles straight into the build, the root's bounds, and
// the largest coordinate for the epsilon. Nothing else of a triangle is kept:
// k_finish_instances makes it again from the mesh, which stays in L2, for
// fewer bytes than writing and gathering it would take.
__global__ void __launch_bounds__(kBuildBlock) k_prepare_instances(Instances in, BuildState st,
                                                                   unsigned long long* __restrict__ max_coord) {
  __shared__ unsigned long long largest;
  if (threadIdx.x == 0) largest = 0;
  __syncthreads();
  float m[12];
  clear_box(m);
  double mc = 0;
  for (int i = blockIdx.x * kBuildBlock + threadIdx.x; i < st.n; i += gridDim.x * kBuildBlock) {
    const int j = instance_of(in, i);
    const DInstance& d = in.inst[j];
    int ids[3];
    double p[9];
    float t[9];
    world_triangle(d, in.meshes[d.mesh], i - in.base[j], ids, p, t);
    for (int q = 0; q < 9; q++) mc = fmax(mc, fabs(p[q]));
    put_prim(st.prims[0], i, t, m);
  }
  for (int off = 16; off > 0; off >>= 1) mc = fmax(mc, __shfl_xor_sync(0xffffffffu, mc, off));
  if ((threadIdx.x & 31) == 0) atomicMax(&largest, static_cast<unsigned long long>(__double_as_longlong(mc)));
  __syncthreads();
  if (threadIdx.x == 0) atomicMax(max_coord, largest);
  put_root_bounds(st, m);
}

// The compiled arrays of instanced geometry in BVH order, for callers that
// keep them (all or none).
struct CompiledArrays {
  float *triangles, *normals, *uvs, *tangents;
  uint32_t* materials;
  uint8_t *flags, *sides;
};

// Every triangle in BVH order, in the render layout (device_scene.cuh): rows of
// vertices with the flag word (the last of a leaf marked from the leaf
// bitmap), material, normals and uvs, tangent; and the vertex bounding box.
// Normals go through the normal matrix and are normalised with Math.hypot, or
// are the face normal. ALL: the compiled arrays too. What bounds it: the latency
// of the double arithmetic and of the mesh reads, so four blocks per SM: 64
// registers and 120 bytes of spills take 1.33 ms for 16.4 M triangles, where 100
// registers (two blocks) took 1.78.
template <bool ALL>
__global__ void __launch_bounds__(kBuildBlock, 4) k_finish_instances(Instances in, BuildState st, PackedGeometry out,
                                                                  CompiledArrays arrays, double* __restrict__ box) {
  VertexBox vb;
  for (int i = blockIdx.x * kBuildBlock + threadIdx.x; i < st.n; i += gridDim.x * kBuildBlock) {
    const int s = static_cast<int>(st.order[i]);
    const int j = instance_of(in, s);
    const DInstance& d = in.inst[j];
    const DMeshRef mr = in.meshes[d.mesh];
    int ids[3];
    double p[9];
    float t[9];
    world_triangle(d, mr, s - in.base[j], ids, p, t);
    float n9[9], u6[6];
    if (mr.nrm && !d.flat) {
      for (int v = 0; v < 3; v++) {
        const float* q = mr.nrm + 3 * static_cast<size_t>(ids[v]);
        const double x = q[0], y = q[1], z = q[2];
        const double nx = d.nm[0] * x + d.nm[3] * y + d.nm[6] * z;
        const double ny = d.nm[1] * x + d.nm[4] * y + d.nm[7] * z;
        const double nz = d.nm[2] * x + d.nm[5] * y + d.nm[8] * z;
        double len = js_hypot3(nx, ny, nz);
        if (!(len != 0) || isnan(len)) len = 1;  // Math.hypot(...) || 1
        n9[3 * v] = static_cast<float>(nx / len);
        n9[3 * v + 1] = static_cast<float>(ny / len);
        n9[3 * v + 2] = static_cast<float>(nz / len);
      }
    } else {
      const double ex = p[3] - p[0], ey = p[4] - p[1], ez = p[5] - p[2];
      const double fx = p[6] - p[0], fy = p[7] - p[1], fz = p[8] - p[2];
      const double cx = ey * fz - ez * fy, cy = ez * fx - ex * fz, cz = ex * fy - ey * fx;
      const double len = js_hypot3(cx, cy, cz);
      float f3[3] = {0.0f, 0.0f, 1.0f};
      if (len > 0) {
        f3[0] = static_cast<float>(cx / len);
        f3[1] = static_cast<float>(cy / len);
        f3[2] = static_cast<float>(cz / len);
      }
      for (int v = 0; v < 3; v++)
        for (int a = 0; a < 3; a++) n9[3 * v + a] = f3[a];
    }
    for (int v = 0; v < 3; v++) {
      u6[2 * v] = mr.uv ? mr.uv[2 * static_cast<size_t>(ids[v])] : 0.0f;
      u6[2 * v + 1] = mr.uv ? mr.uv[2 * static_cast<size_t>(ids[v]) + 1] : 0.0f;
    }
    vb.add(t);
    const float4 tg = tangent_of(t, u6);
    const int next = i + 1;
    const bool last = next == st.n || ((st.leaf_bits[next >> 5] >> (next & 31)) & 1u) != 0;
    const float word = __int_as_float(d.flags | (d.side << 8) | (last ? kLeafEnd : 0));
    const size_t I = static_cast<size_t>(i);
    for (int a = 0; a < 3; a++)
      out.tris[3 * I + a] = make_float4(t[a], static_cast<float>(static_cast<double>(t[a]) + static_cast<double>(t[3 + a])),
                                        static_cast<float>(static_cast<double>(t[a]) + static_cast<double>(t[6 + a])), word);
    out.mats[i] = static_cast<int>(d.material);
    out.attrs[4 * I] = make_float4(n9[0], n9[1], n9[2], n9[3]);
    out.attrs[4 * I + 1] = make_float4(n9[4], n9[5], n9[6], n9[7]);
    out.attrs[4 * I + 2] = make_float4(n9[8], u6[0], u6[1], u6[2]);
    out.attrs[4 * I + 3] = make_float4(u6[3], u6[4], u6[5], 0.0f);
    out.tangents[i] = tg;
    if (ALL) {
      for (int q = 0; q < 9; q++) arrays.triangles[9 * I + q] = t[q];
      for (int q = 0; q < 9; q++) arrays.normals[9 * I + q] = n9[q];
      for (int q = 0; q < 6; q++) arrays.uvs[6 * I + q] = u6[q];
      reinterpret_cast<float4*>(arrays.tangents)[i] = tg;
      arrays.materials[i] = d.material;
      arrays.flags[i] = static_cast<uint8_t>(d.flags);
      arrays.sides[i] = static_cast<uint8_t>(d.side);
    }
  }
  vb.reduce(box);
}

}  // namespace

constexpr int kBuildGrid = 4 * 148;  // blocks of one wave of the level kernels

struct BuildBuffers {
  // build
  DevArray<BuildCtl> ctl;
  DevArray<float4> prim_a[2], prim_b[2];
  DevArray<float2> prim_c[2];
  DevArray<Node> level_nodes[2];
  DevArray<int> segs[2], seg_left, seg_cum;
  DevArray<Acc> acc[2];
  DevArray<Subtree> subtrees;
  DevArray<float4> inner_a, inner_b, leaf_a, leaf_b;
  DevArray<unsigned> inner_t, leaf_t, leaf_bits, depth_bits;
  DevArray<int> rank, scan_sums;
  size_t dirty_words = 0;  // words of depth_bits that the last build may have set
  // compile
  DevArray<double> p, nrm, uv, colors, box;
  DevArray<uint8_t> has_color, flags, sides, flags_out, sides_out;
  DevArray<uint32_t> mats, mats_out, order;
  DevArray<float> tris, tris_out, nrm_out, uv_out, col_out, tan_out, bounds;
  DevArray<int> nodes;
  DevArray<unsigned long long> max_coord;
  // instanced geometry
  DevArray<DInstance> inst;
  DevArray<DMeshRef> mesh_refs;
  DevArray<int> inst_base;
  std::vector<DevArray<float>> mesh_pos, mesh_nrm, mesh_uv;
  std::vector<DevArray<uint32_t>> mesh_idx;
  std::vector<int> mesh_tris;
};

SceneBuilder::SceneBuilder() : b_(new BuildBuffers()) {}
SceneBuilder::~SceneBuilder() { delete b_; }

// The state of a build of n triangles, its buffers made and cleared and its
// root queued; the triangles are the caller's to put in (k_prepare*).
static BuildState start_build(BuildBuffers& B, int n, uint32_t* d_order, int bins, cudaStream_t s) {
  if (bins < 2 || bins > kMaxBins) throw std::runtime_error("bin count out of range");
  const size_t N = static_cast<size_t>(n);
  BuildState st{};
  st.n = n;
  st.words = (n + 31) / 32;
  st.bins = bins;
  // Segments of a level kernel: two waves of blocks over the whole input, so
  // that a small build's upper levels have blocks for every SM.
  const int per_block = (n + 2 * kBuildGrid - 1) / (2 * kBuildGrid);
  st.seg = std::max(kSegMin, std::min(kSegMax, (per_block + kBuildBlock - 1) / kBuildBlock * kBuildBlock));
  // The most nodes of more than kSub triangles that a level can hold, and
  // their segments; every split of one makes at most one more subtree.
  const size_t max_nodes = N / (kSub + 1) + 1;
  const size_t max_segs = N / st.seg + max_nodes;
  const size_t max_subtrees = std::min(N, max_nodes * kBuildDepth + 1);
  const size_t rows = static_cast<size_t>(kBuildDepth) * st.words;
  st.ctl = B.ctl.ensure(1);
  for (int i = 0; i < 2; i++) {
    st.prims[i] = Prims{B.prim_a[i].ensure(N), B.prim_b[i].ensure(N), B.prim_c[i].ensure(N)};
    st.nodes[i] = B.level_nodes[i].ensure(max_nodes);
    st.segs[i] = B.segs[i].ensure(max_segs);
    st.acc[i] = B.acc[i].ensure(N / st.seg + 1);
  }
  st.seg_left = B.seg_left.ensure(max_segs);
  st.seg_cum = B.seg_cum.ensure(max_segs * 3 * kMaxBins);
  st.subtrees = B.subtrees.ensure(max_subtrees);
  st.inner_a = B.inner_a.ensure(N);
  st.inner_b = B.inner_b.ensure(N);
  st.leaf_a = B.leaf_a.ensure(N);
  st.leaf_b = B.leaf_b.ensure(N);
  st.inner_t = B.inner_t.ensure(N);
  st.leaf_t = B.leaf_t.ensure(N);
  st.leaf_bits = B.leaf_bits.ensure(st.words + 1);
  const size_t had = B.depth_bits.n;
  st.depth_bits = B.depth_bits.ensure(rows + kRankGroup);
  if (B.depth_bits.n != had) B.dirty_words = B.depth_bits.n;
  st.rank = B.rank.ensure(rows / kRankGroup + 2);
  st.order = d_order;
  check(cudaMemsetAsync(st.ctl, 0, sizeof(BuildCtl), s), "memset");
  check(cudaMemsetAsync(st.leaf_bits, 0, sizeof(unsigned) * (st.words + 1), s), "memset");
  check(cudaMemsetAsync(st.depth_bits, 0, sizeof(unsigned) * B.dirty_words, s), "memset");
  B.dirty_words = B.depth_bits.n;  // until this build's depth is known
  k_root<<<1, kBuildBlock, 0, s>>>(st);
  return st;
}

// Splits the prepared triangles and numbers the nodes; returns their count
// and, in *levels_out, the levels of the tree.
static int run_build(BuildBuffers& B, const BuildState& st, float* d_bounds, int* d_nodes, int* levels_out,
                     cudaStream_t s) {
  const int n = st.n;
  const size_t N = static_cast<size_t>(n);
  const size_t max_nodes = N / (kSub + 1) + 1;
  int* sums = B.scan_sums.ensure(kScanBlocks);
  // Bin arrays for 16 bins leave room for more warps than those for 32.
  const bool few = st.bins <= 16;
  const auto subtrees = few ? k_subtrees<16> : k_subtrees<kMaxBins>;
  const size_t smem = (few ? sizeof(SubWarp<16>) : sizeof(SubWarp<kMaxBins>)) * kSubWarps;
  check(cudaFuncSetAttribute(subtrees, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)),
        "shared memory");
  // The levels, a few more than a balanced tree has, and the rest of the
  // build behind them; whether that was all is read back once, at the end.
  BuildCtl ctl;
  int levels = 0, want = 0;
  if (n > kSub) {
    while ((static_cast<long long>(kSub) << want) < n) want++;
    want += 4;
  }
  for (;;) {
    want = std::min(want, kBuildDepth);
    for (; levels < want; levels++) {
      const long long most = static_cast<long long>(N / st.seg) +
                             std::min<long long>(max_nodes, levels < 30 ? 1ll << levels : max_nodes);
      // Segments this level has if the tree is balanced, and blocks to suit:
      // smaller ones from four and eight segments per SM. 16.4 M triangles
      // rebuilt and traced 33.8 -> 32.6 ms, 1.3 M 3.82 -> 3.70 (3.81 from 8 and
      // 16 per SM, 3.79 all from 4); with 64 threads at every level, 100 k
      // triangles' hierarchy 0.96 -> 1.01 ms.
      const long long segs = std::max<long long>(
          n / st.seg, std::min<long long>(max_nodes, levels < 30 ? 1ll << levels : max_nodes));
      const int bin_block = segs >= 8 * 148 ? 64 : (segs >= 4 * 148 ? 128 : 256);
      const int part_block = segs >= 4 * 148 ? 128 : 256;
      const auto bin = bin_block == 64 ? k_bin<64> : (bin_block == 128 ? k_bin<128> : k_bin<256>);
      const auto part = part_block == 128 ? k_part<128> : k_part<256>;
      const auto grid = [&](int block) {
        return static_cast<int>(std::min<long long>(most, 2 * kBuildGrid * (kBuildBlock / block)));
      };
      bin<<<grid(bin_block), bin_block, 0, s>>>(levels, st);
      part<<<grid(part_block), part_block, 0, s>>>(levels, st);
    }
    subtrees<<<std::min(blocks_of(n, kSubWarps), 2 * kBuildGrid), 32 * kSubWarps, smem, s>>>(st);
    k_rank_sums<<<kScanBlocks, kScanThreads, 0, s>>>(st, sums);
    k_rank_write<<<kScanBlocks, kScanThreads, 0, s>>>(st, sums);
    k_emit<<<blocks_of(n, 256), 256, 0, s>>>(st, d_bounds, d_nodes);
    check(cudaGetLastError(), "BVH build");
    check(cudaMemcpyAsync(&ctl, st.ctl, sizeof(ctl), cudaMemcpyDeviceToHost, s), "download");
    check(cudaStreamSynchronize(s), "BVH build");
    if (levels >= kBuildDepth || ctl.level[levels].segs == 0) break;
    // A tree with deeper large nodes: more levels, then the subtrees they made.
    check(cudaMemcpyAsync(&st.ctl->next_subtree, &ctl.subtrees, sizeof(int), cudaMemcpyHostToDevice, s), "upload");
    want = levels + 8;
  }
  B.dirty_words = static_cast<size_t>(ctl.inner_depth + 1) * st.words;
  *levels_out = ctl.slot_depth + 1;
  return 1 + 2 * ctl.inner_nodes;
}

namespace {
int prepare_blocks(int n) { return std::min(blocks_of(n, kBuildBlock), 2 * kBuildGrid); }
}  // namespace

int SceneBuilder::build_device(const float* d_tris, int n, float* d_bounds, int* d_nodes, uint32_t* d_order,
                               cudaStream_t s, int bins) {
  last_levels_ = 0;
  if (n <= 0) return 0;
  const BuildState st = start_build(*b_, n, d_order, bins, s);
  k_prepare<<<prepare_blocks(n), kBuildBlock, 0, s>>>(d_tris, st);
  return run_build(*b_, st, d_bounds, d_nodes, &last_levels_, s);
}

void SceneBuilder::upload_meshes(int count, const MeshInput* meshes, cudaStream_t s) {
  BuildBuffers& B = *b_;
  B.mesh_pos.clear();
  B.mesh_nrm.clear();
  B.mesh_uv.clear();
  B.mesh_idx.clear();
  B.mesh_tris.assign(count, 0);
  B.mesh_pos.resize(count);
  B.mesh_nrm.resize(count);
  B.mesh_uv.resize(count);
  B.mesh_idx.resize(count);
  std::vector<DMeshRef> refs(std::max(count, 1));
  auto up = [&](void* d, const void* h, size_t bytes) {
    check(cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, s), "upload");
  };
  for (int i = 0; i < count; i++) {
    const MeshInput& m = meshes[i];
    const size_t v = static_cast<size_t>(m.vertex_count);
    DMeshRef r{};
    r.pos = B.mesh_pos[i].ensure(3 * v);
    up(const_cast<float*>(r.pos), m.position, sizeof(float) * 3 * v);
    if (m.normal) {
      r.nrm = B.mesh_nrm[i].ensure(3 * v);
      up(const_cast<float*>(r.nrm), m.normal, sizeof(float) * 3 * v);
    }
    if (m.uv) {
      r.uv = B.mesh_uv[i].ensure(2 * v);
      up(const_cast<float*>(r.uv), m.uv, sizeof(float) * 2 * v);
    }
    if (m.index_count > 0) {
      r.idx = B.mesh_idx[i].ensure(static_cast<size_t>(m.index_count));
      up(const_cast<uint32_t*>(r.idx), m.index, sizeof(uint32_t) * m.index_count);
    }
    r.tri_count = (m.index_count > 0 ? m.index_count : m.vertex_count) / 3;
    B.mesh_tris[i] = r.tri_count;
    refs[i] = r;
  }
  DMeshRef* d_refs = B.mesh_refs.ensure(refs.size());
  up(d_refs, refs.data(), sizeof(DMeshRef) * refs.size());
  check(cudaStreamSynchronize(s), "mesh upload");
}

long long SceneBuilder::instance_triangles(int count, const InstanceInput* inst) const {
  long long n = 0;
  for (int i = 0; i < count; i++) {
    const int m = inst[i].mesh;
    if (m < 0 || m >= static_cast<int>(b_->mesh_tris.size())) return -1;
    n += b_->mesh_tris[m];
  }
  return n;
}

void SceneBuilder::compile_instances(int count, const InstanceInput* inst, int bins, cudaStream_t s,
                                     const PackedGeometry& packed, bool arrays, DeviceGeometry* out, float* times_ms) {
  BuildBuffers& B = *b_;
  bvh_count_ = -1;
  const long long total = instance_triangles(count, inst);
  if (total < 0) throw std::runtime_error("an instance names a mesh that was not uploaded");
  if (total > (1ll << 30)) throw std::runtime_error("too many triangles");
  const int n = static_cast<int>(total);
  const size_t N = static_cast<size_t>(std::max(n, 1));
  const size_t cap = std::max<size_t>(1, 2 * N - 1);
  cudaEvent_t ev[4];
  for (auto& e : ev) check(cudaEventCreate(&e), "event");
  check(cudaEventRecord(ev[0], s), "event");
  // Instance table: first triangles and words on the host, matrices on the device.
  std::vector<DInstance> h(std::max(count, 1));
  std::vector<int> bases(count + 1, 0);
  for (int i = 0; i < count; i++) {
    DInstance d{};
    std::memcpy(d.world, inst[i].world, sizeof(d.world));
    d.mesh = inst[i].mesh;
    d.flags = inst[i].flags;
    d.side = inst[i].side;
    d.flat = inst[i].flat_shading;
    d.material = inst[i].material;
    bases[i + 1] = bases[i] + B.mesh_tris[d.mesh];
    h[i] = d;
  }
  DInstance* d_inst = B.inst.ensure(h.size());
  int* d_base = B.inst_base.ensure(bases.size());
  check(cudaMemcpyAsync(d_inst, h.data(), sizeof(DInstance) * h.size(), cudaMemcpyHostToDevice, s), "upload");
  check(cudaMemcpyAsync(d_base, bases.data(), sizeof(int) * bases.size(), cudaMemcpyHostToDevice, s), "upload");
  if (count > 0) k_instance_matrices<<<blocks_of(count, 128), 128, 0, s>>>(d_inst, count);
  const Instances in{d_inst, B.mesh_refs.p, d_base, count};
  unsigned long long* d_mc = B.max_coord.ensure(1);
  check(cudaMemsetAsync(d_mc, 0, sizeof(unsigned long long), s), "memset");
  float* d_bounds = B.bounds.ensure(6 * cap);
  int* d_nodes = B.nodes.ensure(3 * cap);
  uint32_t* d_order = B.order.ensure(N);
  last_levels_ = 0;
  int m = 0;
  BuildState st{};
  if (n > 0) {
    st = start_build(B, n, d_order, bins, s);
    k_prepare_instances<<<prepare_blocks(n), kBuildBlock, 0, s>>>(in, st, d_mc);
  }
  check(cudaGetLastError(), "flatten");
  check(cudaEventRecord(ev[1], s), "event");
  if (n > 0) m = run_build(B, st, d_bounds, d_nodes, &last_levels_, s);
  check(cudaEventRecord(ev[2], s), "event");
  DeviceGeometry g{};
  CompiledArrays ca{};
  if (arrays) {
    g.triangles = ca.triangles = B.tris_out.ensure(9 * N);
    g.normals = ca.normals = B.nrm_out.ensure(9 * N);
    g.uvs = ca.uvs = B.uv_out.ensure(6 * N);
    g.tangents = ca.tangents = B.tan_out.ensure(4 * N);
    g.materials = ca.materials = B.mats_out.ensure(N);
    g.flags = ca.flags = B.flags_out.ensure(N);
    g.sides = ca.sides = B.sides_out.ensure(N);
  }
  double box_init[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  double* d_box = B.box.ensure(6);
  check(cudaMemcpyAsync(d_box, box_init, sizeof(box_init), cudaMemcpyHostToDevice, s), "upload");
  if (n > 0) {
    if (arrays) {
      k_finish_instances<true><<<prepare_blocks(n), kBuildBlock, 0, s>>>(in, st, packed, ca, d_box);
    } else {
      k_finish_instances<false><<<prepare_blocks(n), kBuildBlock, 0, s>>>(in, st, packed, ca, d_box);
    }
  }
  check(cudaGetLastError(), "compile");
  double box[6];
  unsigned long long mc_bits = 0;
  check(cudaMemcpyAsync(box, d_box, sizeof(box), cudaMemcpyDeviceToHost, s), "download");
  check(cudaMemcpyAsync(&mc_bits, d_mc, sizeof(mc_bits), cudaMemcpyDeviceToHost, s), "download");
  int root[3] = {0, 0, 0};
  if (m > 0) check(cudaMemcpyAsync(root, d_nodes, sizeof(root), cudaMemcpyDeviceToHost, s), "download");
  check(cudaEventRecord(ev[3], s), "event");
  check(cudaStreamSynchronize(s), "compile");
  double max_coordinate;
  std::memcpy(&max_coordinate, &mc_bits, sizeof(double));
  const double diagonal = n > 0 ? js_hypot3(box[3] - box[0], box[4] - box[1], box[5] - box[2]) : 1.0;
  if (times_ms) {
    for (int i = 0; i < 3; i++) cudaEventElapsedTime(&times_ms[i], ev[i], ev[i + 1]);
  }
  for (auto& e : ev) cudaEventDestroy(e);
  g.n = n;
  g.node_count = m;
  g.root_count = (m > 0 && root[1] > 0) ? root[1] : 0;
  g.epsilon = n > 0 ? std::max(diagonal * 1e-5, std::max(max_coordinate * 2e-6, 1e-7)) : std::max(1e-5, 1e-7);
  g.bounds = d_bounds;
  g.nodes = d_nodes;
  g.order = d_order;
  g.levels = last_levels_;
  *out = g;
}

size_t SceneBuilder::device_bytes() const {
  const BuildBuffers& B = *b_;
  size_t t = B.p.n * 8 + B.nrm.n * 8 +
             B.uv.n * 8 + B.colors.n * 8 + B.tris.n * 4 + B.tris_out.n * 4 + B.nrm_out.n * 4 + B.uv_out.n * 4 +
             B.col_out.n * 4 + B.tan_out.n * 4 + B.bounds.n * 4 + B.nodes.n * 4 + B.mats.n * 4 + B.mats_out.n * 4 +
             B.order.n * 4 + B.flags.n + B.sides.n + B.flags_out.n + B.sides_out.n + B.has_color.n +
             B.inst.n * sizeof(DInstance) + B.inst_base.n * 4 + B.ctl.n * sizeof(BuildCtl) +
             (B.inner_a.n + B.inner_b.n + B.leaf_a.n + B.leaf_b.n) * 16 + (B.inner_t.n + B.leaf_t.n) * 4 +
             (B.leaf_bits.n + B.depth_bits.n + B.rank.n + B.scan_sums.n + B.seg_left.n + B.seg_cum.n) * 4 +
             B.subtrees.n * sizeof(Subtree);
  for (int i = 0; i < 2; i++) {
    t += (B.prim_a[i].n + B.prim_b[i].n) * 16 + B.prim_c[i].n * 8 + B.level_nodes[i].n * sizeof(Node) +
         B.segs[i].n * 4 + B.acc[i].n * sizeof(Acc);
  }
  for (const auto& a : B.mesh_pos) t += a.n * 4;
  for (const auto& a : B.mesh_nrm) t += a.n * 4;
  for (const auto& a : B.mesh_uv) t += a.n * 4;
  for (const auto& a : B.mesh_idx) t += a.n * 4;
  return t;
}

int SceneBuilder::build_bvh_host(const float* tris, int n, cudaStream_t s) {
  bvh_count_ = -1;
  int m = 0;
  if (n > 0) {
    BuildBuffers& B = *b_;
    const size_t N = static_cast<size_t>(n);
    const size_t cap = std::max<size_t>(1, 2 * N - 1);
    float* d_tris = B.tris.ensure(9 * N);
    float* d_bounds = B.bounds.ensure(6 * cap);
    int* d_nodes = B.nodes.ensure(3 * cap);
    uint32_t* d_order = B.order.ensure(N);
    check(cudaMemcpyAsync(d_tris, tris, sizeof(float) * 9 * N, cudaMemcpyHostToDevice, s), "upload");
    m = build_device(d_tris, n, d_bounds, d_nodes, d_order, s);
  }
  bvh_count_ = std::max(n, 0);
  bvh_nodes_ = m;
  return m;
}

bool SceneBuilder::read_bvh(float* bounds, int* nodes, uint32_t* order, cudaStream_t s) {
  if (bvh_count_ < 0) return false;
  if (bvh_count_ == 0) return true;
  BuildBuffers& B = *b_;
  const size_t m = static_cast<size_t>(bvh_nodes_);
  check(cudaMemcpyAsync(bounds, B.bounds.p, sizeof(float) * 6 * m, cudaMemcpyDeviceToHost, s), "download");
  check(cudaMemcpyAsync(nodes, B.nodes.p, sizeof(int) * 3 * m, cudaMemcpyDeviceToHost, s), "download");
  check(cudaMemcpyAsync(order, B.order.p, sizeof(uint32_t) * bvh_count_, cudaMemcpyDeviceToHost, s), "download");
  check(cudaStreamSynchronize(s), "download");
  return true;
}

void SceneBuilder::compile_host(int n, const double* p, const double* nrm, const double* uv, const double* colors,
                                const uint8_t* has_color, const uint32_t* materials, const uint8_t* flags,
                                const uint8_t* sides, float* triangles_out, float* normals_out, float* uvs_out,
                                float* tangents_out, float* colors_out, uint32_t* materials_out, uint8_t* flags_out,
                                uint8_t* sides_out, float* bounds_out, int* nodes_out, uint32_t* order_out,
                                int* node_count_out, double* epsilon_out, int* any_colors, cudaStream_t s) {
  bvh_count_ = -1;
  int any = 0;
  for (int i = 0; i < n && has_color && colors; i++) any |= has_color[i] ? 1 : 0;
  *any_colors = any;
  if (n <= 0) {
    *node_count_out = 0;
    *epsilon_out = 1e-7;  // max(1 * 1e-5, 0, 1e-7) with diagonal 1: compile.ts:388, 401
    *epsilon_out = std::max(1e-5, 1e-7);
    return;
  }
  BuildBuffers& B = *b_;
  const size_t N = static_cast<size_t>(n);
  const size_t cap = std::max<size_t>(1, 2 * N - 1);
  auto up = [&](void* d, const void* h, size_t bytes) {
    check(cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, s), "upload");
  };
  double* d_p = B.p.ensure(9 * N);
  up(d_p, p, sizeof(double) * 9 * N);
  float* d_tris = B.tris.ensure(9 * N);
  unsigned long long* d_mc = B.max_coord.ensure(1);
  check(cudaMemsetAsync(d_mc, 0, sizeof(unsigned long long), s), "memset");
  k_sink_triangles<<<blocks_of(n, 256), 256, 0, s>>>(d_p, n, d_tris, d_mc);
  float* d_bounds = B.bounds.ensure(6 * cap);
  int* d_nodes = B.nodes.ensure(3 * cap);
  uint32_t* d_order = B.order.ensure(N);
  const int m = build_device(d_tris, n, d_bounds, d_nodes, d_order, s);
  double* d_n = B.nrm.ensure(9 * N);
  up(d_n, nrm, sizeof(double) * 9 * N);
  double* d_uv = B.uv.ensure(6 * N);
  up(d_uv, uv, sizeof(double) * 6 * N);
  double* d_col = nullptr;
  uint8_t* d_hc = nullptr;
  if (any) {
    d_col = B.colors.ensure(12 * N);
    up(d_col, colors, sizeof(double) * 12 * N);
    d_hc = B.has_color.ensure(N);
    up(d_hc, has_color, N);
  }
  uint32_t* d_m = B.mats.ensure(N);
  up(d_m, materials, sizeof(uint32_t) * N);
  uint8_t* d_f = B.flags.ensure(N);
  up(d_f, flags, N);
  uint8_t* d_s = B.sides.ensure(N);
  up(d_s, sides, N);
  float* t_out = B.tris_out.ensure(9 * N);
  float* n_out = B.nrm_out.ensure(9 * N);
  float* uv_out = B.uv_out.ensure(6 * N);
  float* c_out = B.col_out.ensure(any ? 12 * N : 1);
  float* tg_out = B.tan_out.ensure(4 * N);
  uint32_t* m_out = B.mats_out.ensure(N);
  uint8_t* f_out = B.flags_out.ensure(N);
  uint8_t* s_out = B.sides_out.ensure(N);
  k_reorder<<<blocks_of(n, 256), 256, 0, s>>>(d_order, n, d_tris, d_n, d_uv, d_col, d_hc, any, d_m, d_f, d_s, t_out,
                                              n_out, uv_out, c_out, m_out, f_out, s_out);
  double box_init[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  double* d_box = B.box.ensure(6);
  up(d_box, box_init, sizeof(box_init));
  k_tangents<<<prepare_blocks(n), kBuildBlock, 0, s>>>(t_out, uv_out, n, reinterpret_cast<float4*>(tg_out), d_box);
  check(cudaGetLastError(), "compile");
  auto down = [&](void* h, const void* d, size_t bytes) {
    check(cudaMemcpyAsync(h, d, bytes, cudaMemcpyDeviceToHost, s), "download");
  };
  down(triangles_out, t_out, sizeof(float) * 9 * N);
  down(normals_out, n_out, sizeof(float) * 9 * N);
  down(uvs_out, uv_out, sizeof(float) * 6 * N);
  down(tangents_out, tg_out, sizeof(float) * 4 * N);
  if (any && colors_out) down(colors_out, c_out, sizeof(float) * 12 * N);
  down(materials_out, m_out, sizeof(uint32_t) * N);
  down(flags_out, f_out, N);
  down(sides_out, s_out, N);
  down(bounds_out, d_bounds, sizeof(float) * 6 * m);
  down(nodes_out, d_nodes, sizeof(int) * 3 * m);
  down(order_out, d_order, sizeof(uint32_t) * N);
  double box[6];
  unsigned long long mc_bits = 0;
  down(box, d_box, sizeof(box));
  down(&mc_bits, d_mc, sizeof(mc_bits));
  check(cudaStreamSynchronize(s), "compile");
  double max_coordinate;
  std::memcpy(&max_coordinate, &mc_bits, sizeof(double));
  const double diagonal = js_hypot3(box[3] - box[0], box[4] - box[1], box[5] - box[2]);
  *node_count_out = m;
  *epsilon_out = std::max(diagonal * 1e-5, std::max(max_coordinate * 2e-6, 1e-7));
}

}  // namespace mcrt
