// BVH traversal on the device.
//
// Triangles are tested with the watertight ray-triangle test of Woop,
// Benthin and Wald (JCGT 2013) in FP32: vertices are translated to the ray
// origin, permuted so the ray's dominant axis is z, and sheared so the ray
// runs along +z; the three 2D edge functions then decide the hit, with a
// double-precision recomputation of any edge function that comes out exactly
// zero. Edge functions are formed without fused multiply-adds so a shared
// edge evaluates to exact negatives in its two triangles. Hits follow the
// reference's rules (src/bvh.ts:226-253): edges inclusive, det == 0 misses,
// FrontSide culls det < 0 and BackSide det > 0, accept 0 < t < t_max.
//
// Boxes are tested with the slab test made conservative as in Ize, "Robust
// BVH Ray Traversal" (JCGT 2013): exit distances are scaled by 1 + 2*gamma(3)
// so rounding can't lose a box a ray grazes, which keeps flat boxes (planes)
// hit as the reference's boxEntry does (src/bvh.ts:340-356).
//
// The walk is the persistent "while-while" traversal of Aila and Laine
// ("Understanding the Efficiency of Ray Traversal on GPUs", HPG 2009, and its
// Kepler/Fermi follow-up): each lane descends inner nodes (nearer child
// first, the other pushed) until every lane of the warp holds a leaf, then
// the warp tests leaves together, which keeps SIMD lanes busy; when enough
// lanes have finished their rays the warp refills them from a global counter
// (dynamic fetch), so a warp never idles waiting on its slowest ray. The
// builder bounds depth at 100, and a deeper foreign tree sets a status bit
// instead of overflowing the stack.
//
// What bounds it: issue slots (60 % busy, half of them on the integer and
// min/max pipe) and the latency of dependent node fetches (L1 65 %, L2 75 %
// hits), at 15-19 active lanes of 32. So the step is kept short: box planes
// and triangle corners go through two-wide float instructions straight from
// the layout (device_scene.cuh), the triangle test's axis permutation is in
// the row addresses, the stack is predicated instead of branched around, each
// lane runs from leaf to leaf on its own, and nothing a walk step reads is in
// local memory. Against scalar tests on component-major nodes with a
// shared-memory short stack inside the query's struct: bounce rays of a
// 1280x720 frame of 500,000 random triangles 5.17 -> 3.98 ms, its shadow rays
// 3.27 -> 2.34 ms (3.83 and 1.95 with the changes noted at walk_step and at
// the shadow queue); shadow rays of the 1.3 M-triangle 1080p frame at 64 passes
// 17.4 -> 13.0 ms (12.3), its closest hits 18.7 -> 16.2 ms (15.8 without the
// making of the camera rays). Every test is the same operations in the same
// rounding, so hits are those of before bit for bit.
//
// Child references: >= 0 an inner node index; < 0 a leaf whose first triangle
// is ~ref. The last triangle of every leaf carries kLeafEnd in its flag word.
#pragma once

#include "device_scene.cuh"

namespace mcrt {

constexpr int kSentinel = 0x7fffffff;  // empty stack / finished ray
constexpr int kRefill = 16;            // refill a warp's finished lanes once this many are idle
// The same threshold for the render's own kernels, measured on the mid workload
// (closest hits: 12, shadow rays: 24, of thresholds between 4 and 32).
constexpr int kRefillClosest = 12;
constexpr int kRefillShadow = 24;

// Status bits a kernel reports back (never a trap).
constexpr unsigned kStatusStackOverflow = 1u;
constexpr unsigned kStatusShadowListOverflow = 2u;
constexpr unsigned kStatusStepLimit = 4u;  // a query hit the step budget and was ended
constexpr unsigned kStatusLeafRange = 8u;  // a leaf ran past the last triangle and was cut

// Node visits plus leaves one query may take: a walk of a well-formed BVH of
// N triangles enters each of its fewer than 2N nodes at most once, so past
// 2N + 64 steps something is wrong and the query ends (kStatusStepLimit)
// instead of looping. A positive sc.step_limit (a test hook) replaces it.
MCRT_D int max_steps(const DScene& sc) { return sc.step_limit > 0 ? sc.step_limit : 2 * sc.tri_count + 64; }

// Two floats in one 64-bit register pair: sm_100a adds, multiplies and fuses
// both halves in one instruction, each half rounded as the scalar
// instruction rounds it, so results are those of the scalar code for half the
// issue slots.
using F2 = unsigned long long;
MCRT_D F2 pack2(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
MCRT_D F2 dup2(float v) { return pack2(v, v); }
MCRT_D float lo2(F2 v) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
  return a;
}
MCRT_D float hi2(F2 v) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
  return b;
}
MCRT_D F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
MCRT_D F2 mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
MCRT_D F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// A ray as the walk uses it: minus the origin and the inverse direction,
// doubled up for the two child boxes, and the triangle test's shear.
struct TravRay {
  F2 nox, noy, noz;  // (-o, -o) per axis
  F2 ivx, ivy, ivz;  // (1 / d, 1 / d) per axis
  float sx, sy;      // shear along the permuted x and y (z's is 1 / d of axis kz)
  int perm;          // kx | ky << 2 | kz << 4: the axes the test permutes to x, y, z
};

MCRT_D float comp(V3 v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : v.z); }

MCRT_D TravRay make_trav_ray(V3 o, V3 d) {
  TravRay r;
  r.nox = dup2(-o.x);
  r.noy = dup2(-o.y);
  r.noz = dup2(-o.z);
  // safeInverse, src/bvh.ts:336-338: a large finite value for a zero component.
  r.ivx = dup2(d.x != 0.0f ? 1.0f / d.x : 1e30f);
  r.ivy = dup2(d.y != 0.0f ? 1.0f / d.y : 1e30f);
  r.ivz = dup2(d.z != 0.0f ? 1.0f / d.z : 1e30f);
  float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
  int kz = (ax >= ay && ax >= az) ? 0 : (ay >= az ? 1 : 2);
  int kx = kz + 1 == 3 ? 0 : kz + 1;
  int ky = kx + 1 == 3 ? 0 : kx + 1;
  float dz = comp(d, kz);
  if (dz < 0.0f) {
    int tmp = kx;
    kx = ky;
    ky = tmp;
  }
  r.perm = kx | (ky << 2) | (kz << 4);
  r.sx = comp(d, kx) / dz;
  r.sy = comp(d, ky) / dz;
  return r;
}

struct TriHit {
  float t, u, v;
  bool front;
};

// What every triangle test of one ray shares, from its TravRay: the permuted
// origin and shear, and the rows of a triangle's three axes.
struct TriFrame {
  F2 nx, ny, nz;     // (-o, -o) along the permuted axes
  F2 nsx, nsy;       // (-sx, -sx), (-sy, -sy)
  float sz;
  int kx, ky, kz;
};

MCRT_D TriFrame make_frame(const TravRay& r) {
  TriFrame f;
  f.kx = r.perm & 3;
  f.ky = (r.perm >> 2) & 3;
  f.kz = r.perm >> 4;
  f.nx = f.kx == 0 ? r.nox : (f.kx == 1 ? r.noy : r.noz);
  f.ny = f.ky == 0 ? r.nox : (f.ky == 1 ? r.noy : r.noz);
  f.nz = f.kz == 0 ? r.nox : (f.kz == 1 ? r.noy : r.noz);
  f.sz = lo2(f.kz == 0 ? r.ivx : (f.kz == 1 ? r.ivy : r.ivz));
  f.nsx = dup2(-r.sx);
  f.nsy = dup2(-r.sy);
  return f;
}

// A triangle's rows along the permuted axes: (v0, v1 | v2, word).
struct TriRows {
  ulonglong2 x, y, z;
  MCRT_D int word() const { return __float_as_int(hi2(x.y)); }
};

MCRT_D TriRows load_rows(const DScene& sc, const TriFrame& f, int k) {
  const ulonglong2* p = reinterpret_cast<const ulonglong2*>(sc.tris) + 3 * static_cast<size_t>(k);
  return TriRows{__ldg(p + f.kx), __ldg(p + f.ky), __ldg(p + f.kz)};
}

// Watertight test of a triangle's rows. cull_side: 0 culls back faces, 1
// culls front faces, anything else culls nothing. Most tests end at the signs
// of the edge functions, which is one branch: the rest (an edge function of
// exactly zero recomputed, the determinant, culling and the distance) is for
// the few that may hit.
MCRT_D bool intersect_triangle(const TriFrame& f, const TriRows& w, float t_max, int cull_side, TriHit& out) {
  const F2 ABz = add2(w.z.x, f.nz);
  const float Ckz = __fadd_rn(lo2(w.z.y), lo2(f.nz));
  const F2 ABx = fma2(f.nsx, ABz, add2(w.x.x, f.nx)), ABy = fma2(f.nsy, ABz, add2(w.y.x, f.ny));
  const float Cx = __fmaf_rn(lo2(f.nsx), Ckz, __fadd_rn(lo2(w.x.y), lo2(f.nx)));
  const float Cy = __fmaf_rn(lo2(f.nsy), Ckz, __fadd_rn(lo2(w.y.y), lo2(f.ny)));
  const float Ax = lo2(ABx), Bx = hi2(ABx), Ay = lo2(ABy), By = hi2(ABy);
  float U = __fsub_rn(__fmul_rn(Cx, By), __fmul_rn(Cy, Bx));
  float V = __fsub_rn(__fmul_rn(Ax, Cy), __fmul_rn(Ay, Cx));
  float W = __fsub_rn(__fmul_rn(Bx, Ay), __fmul_rn(By, Ax));
  const bool zero = fminf(fminf(fabsf(U), fabsf(V)), fabsf(W)) == 0.0f;
  if (fminf(fminf(U, V), W) < 0.0f && fmaxf(fmaxf(U, V), W) > 0.0f && !zero) return false;
  if (zero) {
    U = static_cast<float>(static_cast<double>(Cx) * By - static_cast<double>(Cy) * Bx);
    V = static_cast<float>(static_cast<double>(Ax) * Cy - static_cast<double>(Ay) * Cx);
    W = static_cast<float>(static_cast<double>(Bx) * Ay - static_cast<double>(By) * Ax);
    if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return false;
  }
  const float det = U + V + W;
  if (det == 0.0f) return false;
  if (cull_side == 0 && det < 0.0f) return false;
  if (cull_side == 1 && det > 0.0f) return false;
  const float Az = f.sz * lo2(ABz), Bz = f.sz * hi2(ABz), Cz = f.sz * Ckz;
  const float T = U * Az + V * Bz + W * Cz;
  const float inv = 1.0f / det;
  const float t = T * inv;
  if (!(t > 0.0f && t < t_max)) return false;
  out.t = t;
  out.u = V * inv;
  out.v = W * inv;
  out.front = det > 0.0f;
  return true;
}

// Robust slab test of an inner node's two child boxes: the entry distances
// (>= 0) and whether the ray enters each box before t_max.
struct NodeHit {
  float e0, e1;
  bool h0, h1;
  int left, right;
};

MCRT_D NodeHit test_node(const DNode* nodes, int i, const TravRay& r, float t_max) {
  const float g = 1.0000003576f;  // 1 + 2 * gamma(3) for float
  const ulonglong2* p = reinterpret_cast<const ulonglong2*>(nodes + i);
  const ulonglong2 x = __ldg(p), y = __ldg(p + 1), z = __ldg(p + 2);
  const int2 k = __ldg(reinterpret_cast<const int2*>(p + 3));
  const F2 x0 = mul2(add2(x.x, r.nox), r.ivx), x1 = mul2(add2(x.y, r.nox), r.ivx);
  const F2 y0 = mul2(add2(y.x, r.noy), r.ivy), y1 = mul2(add2(y.y, r.noy), r.ivy);
  const F2 z0 = mul2(add2(z.x, r.noz), r.ivz), z1 = mul2(add2(z.y, r.noz), r.ivz);
  NodeHit n;
  n.e0 = fmaxf(fmaxf(fmaxf(fminf(lo2(x0), lo2(x1)), fminf(lo2(y0), lo2(y1))), fminf(lo2(z0), lo2(z1))), 0.0f);
  n.e1 = fmaxf(fmaxf(fmaxf(fminf(hi2(x0), hi2(x1)), fminf(hi2(y0), hi2(y1))), fminf(hi2(z0), hi2(z1))), 0.0f);
  // Each exit scaled by g, then the least: rounding x * g is monotone in x, so
  // scaling the least exit once gives the same value.
  const float f0 = fminf(fminf(fminf(fmaxf(lo2(x0), lo2(x1)), fmaxf(lo2(y0), lo2(y1))), fmaxf(lo2(z0), lo2(z1))) * g, t_max);
  const float f1 = fminf(fminf(fminf(fmaxf(hi2(x0), hi2(x1)), fmaxf(hi2(y0), hi2(y1))), fmaxf(hi2(z0), hi2(z1))) * g, t_max);
  n.h0 = n.e0 <= f0;
  n.h1 = n.e1 <= f1;
  n.left = k.x;
  n.right = k.y;
  return n;
}

// Traversal stack: the top entry in a register, so that a pop's load is off
// the path to the next node, the entries below it in local memory, one array
// per thread. Pushes and pops are predicated instead of branched around (a
// divergent branch costs the warp three control instructions): a push that is
// not wanted stores nothing, a pop that is not wanted loads nothing. The
// array stands outside the struct: one that is indexed at run time inside it
// would keep the top entry and the address in local memory too.
struct TravStack {
  unsigned at;     // local address of the entry under the top one
  unsigned floor;  // `at` of an empty stack
  int top;         // kSentinel when empty
  // `mem`: kStackMax + 3 ints of the kernel's local memory.
  MCRT_D void init(int* mem) {
    mem[0] = mem[1] = kSentinel;
    floor = static_cast<unsigned>(__cvta_generic_to_local(mem)) + 4u;
    clear();
  }
  MCRT_D void clear() {
    at = floor;
    top = kSentinel;
  }
  // Pushes v if `want`; false if the stack is past its room (and its entries
  // are lost: one comparison against the limit and no branch, since nothing
  // but a report depends on it).
  MCRT_D bool push(int v, bool want) {
    const unsigned limit = floor + 4u * (kStackMax + 1);
    at = min(at + (want ? 4u : 0u), limit);
    asm volatile("{ .reg .pred p; setp.ne.s32 p, %2, 0; @p st.local.s32 [%0], %1; }" ::"r"(at), "r"(top),
                 "r"(static_cast<int>(want))
                 : "memory");
    top = want ? v : top;
    return at != limit;
  }
  // Replaces `node` by the top entry (kSentinel when empty) if `want`. An
  // empty stack may be popped once: that ends its query.
  MCRT_D void pop(int& node, bool want) {
    node = want ? top : node;
    asm volatile("{ .reg .pred p; setp.ne.s32 p, %2, 0; @p ld.local.s32 %0, [%1]; }"
                 : "+r"(top)
                 : "r"(at), "r"(static_cast<int>(want))
                 : "memory");
    at -= want ? 4u : 0u;
  }
};

// A triangle's vertices, flag word and material.
MCRT_D void load_tri(const DScene& sc, int k, V3& a, V3& b, V3& c, int& word, int& material) {
  const float4* p = sc.tris + 3 * static_cast<size_t>(k);
  const float4 x = __ldg(p), y = __ldg(p + 1), z = __ldg(p + 2);
  a = V3{x.x, y.x, z.x};
  b = V3{x.y, y.y, z.y};
  c = V3{x.z, y.z, z.z};
  word = __float_as_int(x.w);
  material = __ldg(sc.tri_mats + k);
}

MCRT_D bool leaf_end(int word) { return (word & kLeafEnd) != 0; }

MCRT_D unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// What a query makes of a triangle it hit (see traverse_persistent).
enum HitAction { kGoOn, kStop, kPause };

// Root reference of the scene: node 0, or the single leaf at triangle 0.
MCRT_D int root_ref(const DScene& sc) { return sc.root_count > 0 ? ~0 : 0; }

// Where one lane's walk stands.
struct WalkState {
  int node = kSentinel;  // next node to visit (kSentinel: none)
  int leaf = 0;          // postponed leaf (< 0), or 0
  int left = 0;          // node visits and leaves the current query may still take, less one
  bool has = false;      // this lane holds an unfinished query
  MCRT_D void start(const DScene& sc) {
    has = true;
    leaf = 0;
    left = max_steps(sc) - 1;
    node = sc.tri_count == 0 ? kSentinel : root_ref(sc);
  }
};

constexpr int kNoSteps = static_cast<int>(0x80000000u);

// One round of every lane's walk: inner nodes until each holds a leaf, then
// leaves; finishes the queries that end. All 32 lanes call it.
template <class Q>
MCRT_D void walk_step(const DScene& sc, Q& q, TravStack& st, WalkState& w, unsigned& status) {
  // A lane may start at, or come back to, a leaf with none postponed.
  {
    const bool take = w.node < 0 && w.leaf == 0;
    w.leaf = take ? w.node : w.leaf;
    st.pop(w.node, take);
  }
  // Descend until every lane holds a leaf (or has finished, or has spent its
  // steps: `left` below zero makes any reference none of an inner node).
  while (static_cast<unsigned>(w.node | (w.left & kNoSteps)) < static_cast<unsigned>(kSentinel)) {
    w.left--;
    const NodeHit h = test_node(sc.nodes, w.node, q.ray(), q.t_max());
    // Nearer child next, the other pushed. The far reference is
    // derived from the near one by xor rather than by a second select
    // on the same condition: nvcc 12.9 at -O1 and above merged such a
    // select pair into one value, pushing the near child twice.
    const int near_ref = (h.h0 && (!h.h1 || h.e0 <= h.e1)) ? h.left : h.right;
    if (!st.push(h.left ^ h.right ^ near_ref, h.h0 && h.h1)) status |= kStatusStackOverflow;
    // A leaf is postponed and the walk goes on with the top entry, as it does
    // where neither box is entered. One pop for both; a popped leaf waits for
    // the end of the descent. Two pops, the second for a popped leaf, took
    // five instructions more a visit and waited for the first one's load: with
    // this, and the step budget in the loop's own condition, 500 k unstructured
    // triangles at 720p 5.81 -> 5.64 ms a frame, the mid scene at 1080p 37.2 ->
    // 36.6, 16.4 M instanced triangles' trace 10.2 -> 9.7. (Leaving the descent
    // once all but 1, 3 or 8 lanes hold a leaf: 2, 5 and 13 % slower on the soup;
    // never leaving it early: 4 %; lanes that hold a leaf waiting there: 19 %.)
    const bool any = h.h0 || h.h1;
    const bool take = any && near_ref < 0 && w.leaf == 0;
    w.leaf = take ? near_ref : w.leaf;
    w.node = near_ref;
    st.pop(w.node, take || !any);
    if (!__any_sync(__activemask(), w.leaf == 0)) break;
  }
  {
    const bool take = w.node < 0 && w.leaf == 0;
    w.leaf = take ? w.node : w.leaf;
    st.pop(w.node, take);
  }
  // Test the postponed leaf, then any leaf reached right after it, each
  // lane going on to its next triangle on its own.
  bool stop = false, paused = false;
  if (w.leaf < 0 && w.left >= 0) {
    w.left--;
    const TriFrame f = make_frame(q.ray());
    int k = ~w.leaf;
    for (;;) {
      const TriRows rows = load_rows(sc, f, k);
      const bool end = leaf_end(rows.word()) || k + 1 >= sc.tri_count;
      TriHit th;
      if (intersect_triangle(f, rows, q.t_max(), q.side(rows.word()), th)) {
        const HitAction a = q.hit(k, th, rows.word());
        stop = a == kStop;
        paused = a == kPause;
        if (a != kGoOn) {
          w.leaf = end ? 0 : ~(k + 1);  // the rest of the leaf, for a pause
          w.left += end ? 0 : 1;        // which is no further step
          break;
        }
      }
      k++;
      if (end) {
        w.leaf = 0;
        if (w.node >= 0) break;
        w.leaf = w.node;
        k = ~w.node;
        st.pop(w.node, true);
        if (w.left < 0) break;
        w.left--;
      }
    }
  }
  if (paused) stop = !q.resume();
  if (stop) {
    w.node = kSentinel;
    w.leaf = 0;
  }
  // Out of steps with something left to visit (a query that its last step ended is none).
  if (w.left < 0 && (w.node != kSentinel || w.leaf != 0)) {
    status |= kStatusStepLimit;
    w.node = kSentinel;
    w.leaf = 0;
  }
  if (w.has && w.node == kSentinel && w.leaf == 0) {
    q.finish();
    w.has = false;
    w.left = 0;
  }
}

// Persistent while-while traversal of queries [0, n) for one warp, taking
// work from *counter. Q supplies, per lane:
//   void load(int index)      start query `index` (ray, limits, result state)
//   const TravRay& ray()
//   float t_max()             current upper limit (closest hit lowers it)
//   int side(int word)        the triangle test's cull_side
//   HitAction hit(int k, const TriHit& h, int word)  triangle k is hit:
//                             kStop ends the query (any hit: blocked), kPause
//                             asks for resume() before the next triangle
//   bool resume()             the answer to a pause; false ends the query
//   void finish()             write the query's result
// REFILL: a warp takes new queries once that many of its lanes are idle.
// lanes: how many lanes of each warp take queries (query_lanes).
//
// With few queries (a wavefront's last bounces, a tile, a handful of picking
// rays) a full warp per 32 of them would leave most of the GPU idle while each
// warp steps through the union of its lanes' walks, so the queries are spread
// over the resident warps: a power of two of them per warp. One query per warp
// while there are warps for it measured best of one to 64 queries per resident
// warp: a 64 x 64 tile's closest hits 0.17 -> 0.13 ms and shadow rays 0.15 ->
// 0.12 ms over its bounces, and no difference once the GPU is full.
MCRT_D int query_lanes(int n) {
  const unsigned warps = gridDim.x * (blockDim.x >> 5);
  const unsigned per = (static_cast<unsigned>(n) + warps - 1) / warps;
  return per >= 17u ? 32 : (per <= 1u ? 1 : 1 << (32 - __clz(per - 1)));
}

template <int REFILL = kRefill, class Q>
MCRT_D void traverse_persistent(const DScene& sc, Q& q, int n, int lanes, unsigned* counter, TravStack& st,
                                unsigned& status) {
  const unsigned lane = threadIdx.x & 31;
  WalkState w;
  bool exhausted = static_cast<int>(lane) >= lanes;
  const int refill = 32 - lanes + max(1, REFILL * lanes / 32);  // lanes without a query that call for a refill
  for (;;) {
    // Refill finished lanes with one atomic per warp.
    const bool need = !w.has && !exhausted;
    const unsigned mneed = __ballot_sync(0xffffffffu, need);
    if (mneed) {
      const int leader = __ffs(mneed) - 1;
      unsigned base = 0;
      if (static_cast<int>(lane) == leader) base = atomicAdd(counter, __popc(mneed));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (need) {
        const unsigned idx = base + __popc(mneed & lanemask_lt());
        if (idx < static_cast<unsigned>(n)) {
          q.load(static_cast<int>(idx));
          st.clear();
          w.start(sc);
        } else {
          exhausted = true;
        }
      }
    }
    if (__all_sync(0xffffffffu, !w.has)) return;  // every lane is exhausted
    do {
      walk_step(sc, q, st, w, status);
    } while (__popc(__ballot_sync(0xffffffffu, !w.has)) < refill && __any_sync(0xffffffffu, w.has));
  }
}

// Warp-coherent traversal of queries [0, n): each warp takes 32 consecutive
// queries and walks the union of their paths through the tree together, one
// node at a time, every lane testing that node's child boxes against its own
// ray (the node is one broadcast load). A child is entered with the lanes
// whose ray enters its box, first the child most of those lanes reach first;
// the other is pushed with its lane mask on a warp stack in shared memory
// (`stack`, kStackMax entries, written by every lane with the same value).
// Each lane thus visits exactly the nodes its own box tests admit, with the
// same closest hit or blocking result as the per-lane walk; only the order
// among a lane's subtrees can differ, which matters for hits at exactly equal
// distance. With no divergence the warp runs at full width, which pays for
// rays that share most of their paths and all run to the end: camera rays,
// where a warp holds the passes of one or two pixels. Q is the same query
// interface as traverse_persistent's, for closest hits (no leaf ends them).
template <class Q>
MCRT_D void traverse_packet(const DScene& sc, Q& q, int n, unsigned* counter, int2* stack, unsigned& status) {
  const unsigned lane = threadIdx.x & 31;
  const unsigned bit = 1u << lane;
  const int step_limit = max_steps(sc);
  for (;;) {
    unsigned base = 0;
    if (lane == 0) base = atomicAdd(counter, 32u);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base >= static_cast<unsigned>(n)) return;
    const bool has = base + lane < static_cast<unsigned>(n);
    if (has) q.load(static_cast<int>(base + lane));
    const unsigned live = __ballot_sync(0xffffffffu, has);
    int node = sc.tri_count == 0 ? kSentinel : root_ref(sc);
    unsigned mask = live;
    int sp = 0;
    int steps = 0;
    while (node != kSentinel && live != 0) {
      if (mask != 0) {
        if (++steps > step_limit) {
          if (live & bit) status |= kStatusStepLimit;
          break;
        }
        if (node >= 0) {
          // Every lane tests; a lane outside the mask, or without a query, is masked out of the votes.
          const NodeHit nd = test_node(sc.nodes, node, q.ray(), q.t_max());
          const unsigned m0 = __ballot_sync(0xffffffffu, nd.h0) & mask, m1 = __ballot_sync(0xffffffffu, nd.h1) & mask;
          if (m0 != 0 && m1 != 0) {
            const unsigned first_left = __ballot_sync(0xffffffffu, nd.h0 && (!nd.h1 || nd.e0 <= nd.e1)) & mask;
            const bool left = 2 * __popc(first_left) >= __popc(m0 | m1);
            if (sp < kStackMax) {
              stack[sp] = left ? make_int2(nd.right, static_cast<int>(m1)) : make_int2(nd.left, static_cast<int>(m0));
              sp++;
            } else if (live & bit) {
              status |= kStatusStackOverflow;
            }
            node = left ? nd.left : nd.right;
            mask = left ? m0 : m1;
            continue;
          }
          if (m0 != 0 || m1 != 0) {
            node = m0 != 0 ? nd.left : nd.right;
            mask = m0 | m1;
            continue;
          }
        } else {
          if (mask & bit) {
            const TriFrame f = make_frame(q.ray());
            for (int k = ~node; k < sc.tri_count; k++) {
              const TriRows rows = load_rows(sc, f, k);
              TriHit th;
              // Closest hits never stop at one.
              if (intersect_triangle(f, rows, q.t_max(), q.side(rows.word()), th)) q.hit(k, th, rows.word());
              if (leaf_end(rows.word())) break;
            }
          }
        }
      }
      if (sp == 0) break;
      --sp;
      const int2 e = stack[sp];
      node = e.x;
      mask = static_cast<unsigned>(e.y);
    }
    if (has) q.finish();
  }
}

// Closest hit of one query: intersectClosest, src/bvh.ts:202-282.
struct ClosestState {
  TravRay r;
  float tmax;      // the closest hit's distance (infinity: none)
  float u, v;
  unsigned hit;    // (front << 31) | (triangle + 1), or 0
  bool cull;
  MCRT_D void start(V3 o, V3 d, bool c) {
    r = make_trav_ray(o, d);
    tmax = __int_as_float(0x7f800000);
    cull = c;
    u = v = 0.0f;
    hit = 0u;
  }
  MCRT_D int triangle() const { return static_cast<int>(hit & 0x7fffffffu) - 1; }
  MCRT_D float t() const { return hit != 0u ? tmax : 0.0f; }
  MCRT_D int cull_side(int word) const { return cull ? tri_side(word) : 2; }
  MCRT_D void take(int k, const TriHit& h) {
    tmax = h.t;
    u = h.u;
    v = h.v;
    hit = (h.front ? 0x80000000u : 0u) | static_cast<unsigned>(k + 1);
  }
};

}  // namespace mcrt
