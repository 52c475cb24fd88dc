// pk_bvh_sweep.cu -- GPU rebuild of the reference BVH: bvh.js full-sweep object
// SAH (render/bvh.js:12-223, render/primitives.js:3-44), BFS serialisation
// (bvh.js:46-74) and trace_pass.js packing (trace_pass.js:166-170,202-262).
//
// Exactness.  Every reference ref list of a node is its triangles ordered by
// (centroid[axis], triangle index): the root lists come from a stable sort of
// triangles in index order, and #splitNode keeps relative order.  Here each
// node owns one range of positions in three arrays (one per axis) that hold
// exactly those lists, partitioned in place level by level.
//   The sweep cost of position i of a node of n triangles is
//     0.5 + (SA(prefix) / SA(node)) (i + 1) + (SA(suffix) / SA(node)) (n - 1 - i)
// (bvh.js:195-208, suffix from i on), in double, and the first minimum in
// (axis, index) order wins.  FP64 runs at two lanes per clock and SM here, so
// evaluating all 3 n costs of a level in double was most of the old build
// (20 of 31 ms of kernels for 1.3M triangles, 177 FP64 operations per
// triangle and level).  Instead the boxes are scanned in binary32 (rounding a
// coordinate is monotone, so the union of rounded boxes is the rounded union),
// every cost is computed in binary32 with a bound E on its distance from the
// double cost, and only the costs within 2E of the smallest are evaluated
// again in double from exact boxes: any other cost is certainly larger.
//   Exact boxes are kept as order-preserving 64-bit integers (a double's bits
// with the lower 63 flipped when negative), so their unions are integer
// minima and maxima.
//
// Two phases.  Nodes of more than SUB triangles are split one level per round
// over tiles of the whole array (k_lv_*).  A node of at most SUB triangles is
// finished by one block in shared memory (k_subtree), all its levels in one
// launch; the old build ran every one of its 26 levels over all triangles in
// memory.  A node's BFS index and a leaf's first triangle then follow from
// per-level counts of the subtrees, summed from left to right (k_columns).
//   1,310,730 triangles, whole build: 41.1 ms level by level, 8.0 in two phases,
// 7.5 with the subtrees' scans in one copy (k_subtree).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "pk_bvh.h"
#include "pk_bvh_pack.cuh"
#include "pk_internal.cuh"
#include "pk_util.h"

namespace pk {
namespace {

typedef long long i64;
typedef unsigned long long u64;

constexpr i64 KEY_MAX = 0x7fffffffffffffffll;

__device__ __forceinline__ i64 key_of(double x) {
  const i64 b = __double_as_longlong(x);
  return b ^ ((b >> 63) & KEY_MAX);
}
__device__ __forceinline__ double val_of(i64 k) { return __longlong_as_double(k ^ ((k >> 63) & KEY_MAX)); }

struct KBox {  // exact box as ordered keys
  i64 mn[3], mx[3];
};
__device__ __forceinline__ KBox kbox_empty() {
  KBox b;
#pragma unroll
  for (int a = 0; a < 3; a++) { b.mn[a] = KEY_MAX; b.mx[a] = -KEY_MAX - 1; }
  return b;
}
__device__ __forceinline__ void kbox_add(KBox& a, const KBox& b) {
#pragma unroll
  for (int i = 0; i < 3; i++) {
    a.mn[i] = b.mn[i] < a.mn[i] ? b.mn[i] : a.mn[i];
    a.mx[i] = b.mx[i] > a.mx[i] ? b.mx[i] : a.mx[i];
  }
}
__device__ __forceinline__ KBox kbox_shfl_xor(const KBox& b, int o) {
  KBox r;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    r.mn[i] = __shfl_xor_sync(0xffffffffu, b.mn[i], o);
    r.mx[i] = __shfl_xor_sync(0xffffffffu, b.mx[i], o);
  }
  return r;
}
template <bool REV>
__device__ __forceinline__ KBox kbox_shfl_from(const KBox& b, int o) {  // from the lane o earlier in scan order
  KBox r;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    r.mn[i] = REV ? __shfl_down_sync(0xffffffffu, b.mn[i], o) : __shfl_up_sync(0xffffffffu, b.mn[i], o);
    r.mx[i] = REV ? __shfl_down_sync(0xffffffffu, b.mx[i], o) : __shfl_up_sync(0xffffffffu, b.mx[i], o);
  }
  return r;
}
__device__ __forceinline__ void kbox_warp(KBox& b) {
#pragma unroll
  for (int o = 16; o; o >>= 1) kbox_add(b, kbox_shfl_xor(b, o));
}
// BoundingBox.getSurfaceArea (primitives.js:39-44)
__device__ __forceinline__ double kbox_sa(const KBox& b) {
  const double xl = fmax(val_of(b.mx[0]) - val_of(b.mn[0]), 0.0);
  const double yl = fmax(val_of(b.mx[1]) - val_of(b.mn[1]), 0.0);
  const double zl = fmax(val_of(b.mx[2]) - val_of(b.mn[2]), 0.0);
  return (xl * yl + xl * zl + yl * zl) * 2.0;
}
// bvh.js:195-208
__device__ __forceinline__ double sweep_cost(double saf, double sab, double psa, uint32_t i, uint32_t n) {
  return 0.5 + (saf / psa) * (double)(i + 1) + (sab / psa) * (double)(n - 1 - i);
}

// Rounded box: binary32 coordinates in [0, 1] of a frame that holds the box
// (non-negative, so their bits order as unsigned integers).
struct FBox {
  uint32_t mn[3], mx[3];
};
__device__ __forceinline__ FBox fbox_empty() {
  FBox b;
#pragma unroll
  for (int a = 0; a < 3; a++) { b.mn[a] = 0xffffffffu; b.mx[a] = 0u; }
  return b;
}
__device__ __forceinline__ void fbox_add(FBox& a, const FBox& b) {
#pragma unroll
  for (int i = 0; i < 3; i++) { a.mn[i] = min(a.mn[i], b.mn[i]); a.mx[i] = max(a.mx[i], b.mx[i]); }
}
template <bool REV>
__device__ __forceinline__ FBox fbox_shfl_from(const FBox& b, int o) {
  FBox r;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    r.mn[i] = REV ? __shfl_down_sync(0xffffffffu, b.mn[i], o) : __shfl_up_sync(0xffffffffu, b.mn[i], o);
    r.mx[i] = REV ? __shfl_down_sync(0xffffffffu, b.mx[i], o) : __shfl_up_sync(0xffffffffu, b.mx[i], o);
  }
  return r;
}
__device__ __forceinline__ void fbox_warp(FBox& b) {
#pragma unroll
  for (int i = 0; i < 3; i++) {
    b.mn[i] = __reduce_min_sync(0xffffffffu, b.mn[i]);
    b.mx[i] = __reduce_max_sync(0xffffffffu, b.mx[i]);
  }
}
__device__ __forceinline__ float fbox_ext(const FBox& b, int a) {
  return __uint_as_float(b.mx[a]) - __uint_as_float(b.mn[a]);
}
__device__ __forceinline__ float fbox_sa(const FBox& b) {
  const float x = fbox_ext(b, 0), y = fbox_ext(b, 1), z = fbox_ext(b, 2);
  return (x * y + x * z + y * z) * 2.0f;
}
__device__ __forceinline__ uint32_t rounded(double v, double lo, double scale) {
  return __float_as_uint(__double2float_rn((v - lo) * scale));
}

// Frame of a box: lower corner and a power of two that maps its largest extent
// into (1/2, 1]; unusable (every cost then evaluated in double) when the double
// areas may leave the normal numbers.  cost_bound accepts areas down to 2^-40 of
// the squared extent: from 1e-140 on they are normal and what underflows in the
// areas inside them is below 1e-20 of them; up to 1e150 sums of products stay finite.
struct Frame {
  double lo[3], scale;
  bool ok;
};
__device__ __forceinline__ Frame frame_of(const KBox& b) {
  Frame f;
  double ext = 0.0;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    f.lo[a] = val_of(b.mn[a]);
    ext = fmax(ext, val_of(b.mx[a]) - f.lo[a]);
  }
  f.ok = ext > 1e-140 && ext < 1e150;
  int e = 0;
  if (f.ok) frexp(ext, &e);
  f.scale = f.ok ? ldexp(1.0, -e) : 0.0;
  return f;
}

// Bound on |binary32 cost - double cost| of any position of a node, from its
// rounded box.  Coordinates are off by at most 2^-24 (they are at most 1), so
// an extent by at most 3 * 2^-24 < e with its own rounding; an area of a box
// inside the node by at most 4 e (X + Y + Z) + 6 e^2 plus 2^-21 of the node's
// for its operations (A below, doubled there); a quotient of areas by 2 A / P,
// a cost by 2 n A / P plus 2^-21 n for its operations.  Returned at twice
// that; infinite when A is not small against P, and then every position is
// evaluated in double.
__device__ __forceinline__ float cost_bound(const FBox& b, uint32_t n, bool ok) {
  const float e = 0x1p-22f;
  const float P = fbox_sa(b);
  const float A = 4.0f * e * (fbox_ext(b, 0) + fbox_ext(b, 1) + fbox_ext(b, 2)) + 6.0f * e * e + 0x1p-20f * P;
  if (!ok || !(P > 16.0f * A)) return __int_as_float(0x7f800000);
  return (float)n * (4.0f * A / P + 0x1p-20f);
}

__device__ __forceinline__ KBox load_kbox(const KBox* p) {
  const longlong2* q = reinterpret_cast<const longlong2*>(p);
  const longlong2 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
  KBox r;
  r.mn[0] = a.x; r.mn[1] = a.y; r.mn[2] = b.x;
  r.mx[0] = b.y; r.mx[1] = c.x; r.mx[2] = c.y;
  return r;
}

// ---- per-triangle boxes, sort keys (Node.sortRefs) and the root box ---------------
constexpr int TRI_THREADS = 256;
__global__ void __launch_bounds__(TRI_THREADS) k_tri_boxes(const double* __restrict__ pos3,
                                                           const int4* __restrict__ tri4, uint32_t n,
                                                           KBox* __restrict__ boxes, u64* __restrict__ keys,
                                                           uint32_t* __restrict__ vals, KBox* __restrict__ root) {
  __shared__ KBox s_box[TRI_THREADS / 32];
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  KBox kb = kbox_empty();
  if (t < n) {
    const int4 tr = tri4[t];
    const int v[3] = {tr.x, tr.y, tr.z};
    double mn[3], mx[3];
#pragma unroll
    for (int a = 0; a < 3; a++) { mn[a] = __longlong_as_double(0x7ff0000000000000ll); mx[a] = -mn[a]; }
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const double* p = pos3 + 3 * (size_t)v[k];
#pragma unroll
      for (int a = 0; a < 3; a++) { mn[a] = fmin(p[a], mn[a]); mx[a] = fmax(p[a], mx[a]); }
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
      kb.mn[a] = key_of(mn[a]);
      kb.mx[a] = key_of(mx[a]);
      double c = (mn[a] + mx[a]) * 0.5;  // BoundingBox.centroid (primitives.js:32-37)
      if (c == 0.0) c = 0.0;             // -0 and +0 compare equal in the reference sort
      const u64 u = (u64)__double_as_longlong(c);
      keys[(size_t)a * n + t] = (u >> 63) ? ~u : (u | 0x8000000000000000ull);
      vals[(size_t)a * n + t] = t;
    }
    boxes[t] = kb;
  }
  kbox_warp(kb);
  if ((threadIdx.x & 31) == 0) s_box[threadIdx.x >> 5] = kb;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < TRI_THREADS / 32; w++) kbox_add(kb, s_box[w]);
    for (int a = 0; a < 3; a++) {
      atomicMin(&root->mn[a], kb.mn[a]);
      atomicMax(&root->mx[a], kb.mx[a]);
    }
  }
}

// Control words of a build.
struct Ctl {
  KBox root;
  Frame frame;                // of the root
  uint32_t n_nodes, n_tiles;  // of the level in hand
  uint32_t n_small, n_big;    // subtrees so far, large nodes so far
  uint32_t inner;             // inner nodes inside subtrees
  uint32_t levels;            // deepest level + 1
  uint32_t err, pad;
};
__global__ void k_init(Ctl* c) {
  c->root = kbox_empty();
  c->n_nodes = c->n_tiles = c->n_small = c->n_big = c->inner = c->levels = c->err = 0u;
}

__global__ void k_frame(Ctl* c) { c->frame = frame_of(c->root); }

// Rounded boxes in the root's frame: {min xyz, max x}{max yz, -, -}.
__global__ void k_round_boxes(const KBox* __restrict__ boxes, uint32_t n, const Ctl* __restrict__ ctl,
                              uint4* __restrict__ fb) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const Frame f = ctl->frame;
  const KBox k = load_kbox(boxes + t);
  uint32_t r[6];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    r[a] = rounded(val_of(k.mn[a]), f.lo[a], f.scale);
    r[3 + a] = rounded(val_of(k.mx[a]), f.lo[a], f.scale);
  }
  fb[2 * (size_t)t] = make_uint4(r[0], r[1], r[2], r[3]);
  fb[2 * (size_t)t + 1] = make_uint4(r[4], r[5], 0u, 0u);
}
__device__ __forceinline__ FBox load_fbox(const uint4* fb, uint32_t t) {
  const uint4 a = __ldg(fb + 2 * (size_t)t);
  const uint2 b = __ldg(reinterpret_cast<const uint2*>(fb + 2 * (size_t)t + 1));
  FBox r;
  r.mn[0] = a.x; r.mn[1] = a.y; r.mn[2] = a.z;
  r.mx[0] = a.w; r.mx[1] = b.x; r.mx[2] = b.y;
  return r;
}

// =====================================================================
// Phase 1: large nodes, one level per round.  Work items are (axis, tile)
// pairs; a tile lies inside one node.
// =====================================================================
constexpr uint32_t SUB = 512;  // triangles a block finishes by itself
constexpr int LV_THREADS = 256;
constexpr int LV_ITEMS = 4;
constexpr uint32_t LV_TILE = LV_THREADS * LV_ITEMS;
constexpr int LV_WARPS = LV_THREADS / 32;

struct LNode {
  uint32_t start, count, tile0, ntiles;
};
struct LTile {
  uint32_t node, off;
};
struct SmallTask {
  uint32_t start, count, level, buf;  // buf: which of the two list arrays holds its range
};
struct Best {
  double cost;
  uint32_t key, pad;  // axis * count + index; ~0: none
};

struct Level {
  Ctl* ctl;
  const KBox* kbox;
  const uint4* fbox;
  int32_t* A[2];       // lists [3][T], ping-pong by level
  uint32_t T, max_tiles;
  LNode* node[2];
  LTile* tile[2];
  FBox* tbox;          // [3][max_tiles] boxes of tiles
  FBox* carry[2];      // [3][max_tiles] union of the node's tiles before / after
  KBox* etbox;
  KBox* ecarry[2];
  FBox* nbox;          // per node
  uint32_t* nmin;      // [node][3] smallest binary32 cost (bits)
  uint32_t* tmin;      // [3][max_tiles]
  float* cost;         // [3][T]
  KBox* nexact;        // per node
  Best* best;          // [3][max_tiles]
  uint32_t* split;     // per node: axis
  uint32_t* nleft;
  uint32_t* tcount;    // [3][max_tiles] left triangles of a tile, then the node's before it
  uint8_t* left;       // per triangle
  uint32_t* big_start;
  KBox* big_box;
  uint32_t* big_off;   // per level: large nodes before it (big_off[d + 1] - big_off[d] of them)
  SmallTask* small;
};

__device__ __forceinline__ float lv_limit(const Level& L, uint32_t k, uint32_t count) {
  const uint32_t m = min(min(L.nmin[3 * k], L.nmin[3 * k + 1]), L.nmin[3 * k + 2]);
  return __uint_as_float(m) + 2.0f * cost_bound(L.nbox[k], count, L.ctl->frame.ok);
}
__device__ __forceinline__ bool beyond(uint32_t cost_bits, float limit) { return __uint_as_float(cost_bits) > limit; }

// The root alone.  After a failed sort the lists hold no triangle numbers: no
// nodes and no tiles then, so that no kernel of any level reads them.
__global__ void k_lv_start(Level L, uint32_t T) {
  const uint32_t nt = (T + LV_TILE - 1) / LV_TILE;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const bool ok = L.ctl->err == 0u;
    L.node[0][0] = LNode{0u, T, 0u, nt};
    L.ctl->n_nodes = ok ? 1u : 0u;
    L.ctl->n_tiles = ok ? nt : 0u;
    L.big_off[0] = 0;
  }
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < nt; t += gridDim.x * blockDim.x)
    L.tile[0][t] = LTile{0u, t * LV_TILE};
}

__global__ void __launch_bounds__(LV_THREADS) k_lv_reduce(Level L, int b) {
  __shared__ FBox s_box[LV_WARPS];
  const uint32_t nt = L.ctl->n_tiles;
  for (uint32_t w = blockIdx.x; w < 3 * nt; w += gridDim.x) {
    const uint32_t axis = w / nt, t = w % nt;
    const LTile tl = L.tile[b][t];
    const LNode nd = L.node[b][tl.node];
    const uint32_t n = min(LV_TILE, nd.count - tl.off);
    const int32_t* A = L.A[b] + (size_t)axis * L.T + nd.start + tl.off;
    FBox bx = fbox_empty();
    for (uint32_t i = threadIdx.x; i < n; i += LV_THREADS) fbox_add(bx, load_fbox(L.fbox, (uint32_t)A[i]));
    fbox_warp(bx);
    if ((threadIdx.x & 31) == 0) s_box[threadIdx.x >> 5] = bx;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int k = 1; k < LV_WARPS; k++) fbox_add(bx, s_box[k]);
      L.tbox[(size_t)axis * L.max_tiles + t] = bx;
    }
    __syncthreads();
  }
}

// One warp per (node, axis): the unions of the node's tiles before and after each.
template <bool REV>
__device__ __forceinline__ FBox lv_carry(const FBox* in, FBox* out, uint32_t n, int lane) {
  FBox run = fbox_empty();
  for (uint32_t base = 0; base < n; base += 32) {
    const uint32_t i = base + (uint32_t)lane;
    FBox v = i < n ? in[REV ? n - 1 - i : i] : fbox_empty();
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const FBox u = fbox_shfl_from<false>(v, o);
      if (lane >= o) fbox_add(v, u);
    }
    FBox ex = fbox_shfl_from<false>(v, 1);
    if (lane == 0) ex = fbox_empty();
    fbox_add(ex, run);
    if (i < n) out[REV ? n - 1 - i : i] = ex;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      run.mn[a] = min(run.mn[a], __shfl_sync(0xffffffffu, v.mn[a], 31));
      run.mx[a] = max(run.mx[a], __shfl_sync(0xffffffffu, v.mx[a], 31));
    }
  }
  return run;
}
__global__ void __launch_bounds__(LV_THREADS) k_lv_carry(Level L, int b) {
  const int lane = threadIdx.x & 31;
  const uint32_t items = 3 * L.ctl->n_nodes;
  for (uint32_t w = (blockIdx.x * LV_THREADS + threadIdx.x) >> 5; w < items; w += (gridDim.x * LV_THREADS) >> 5) {
    const uint32_t k = w / 3, axis = w % 3;
    const LNode nd = L.node[b][k];
    const size_t o = (size_t)axis * L.max_tiles + nd.tile0;
    const FBox all = lv_carry<false>(L.tbox + o, L.carry[0] + o, nd.ntiles, lane);
    lv_carry<true>(L.tbox + o, L.carry[1] + o, nd.ntiles, lane);
    if (lane == 0) {
      L.nmin[w] = 0xffffffffu;
      if (axis == 0) L.nbox[k] = all;
    }
  }
}

// Running unions of a tile in list order (REV: from its end), including the
// carry: calls f(j, box) for this thread's LV_ITEMS consecutive positions.
template <bool REV, class F>
__device__ __forceinline__ void tile_scan(const FBox (&bx)[LV_ITEMS], const FBox& carry, FBox* s_warp, F f) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  FBox inc = bx[0];
#pragma unroll
  for (int j = 1; j < LV_ITEMS; j++) fbox_add(inc, bx[j]);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const FBox u = fbox_shfl_from<REV>(inc, o);
    if (REV ? lane + o < 32 : lane >= o) fbox_add(inc, u);
  }
  if (lane == (REV ? 0 : 31)) s_warp[warp] = inc;
  __syncthreads();
  FBox run = fbox_shfl_from<REV>(inc, 1);
  if (lane == (REV ? 31 : 0)) run = fbox_empty();
  fbox_add(run, carry);
  for (int k = 0; k < LV_WARPS; k++)
    if (REV ? k > warp : k < warp) fbox_add(run, s_warp[k]);
#pragma unroll
  for (int q = 0; q < LV_ITEMS; q++) {
    const int j = REV ? LV_ITEMS - 1 - q : q;
    fbox_add(run, bx[j]);
    f(j, run);
  }
}

__global__ void __launch_bounds__(LV_THREADS) k_lv_cost(Level L, int b) {
  __shared__ FBox s_fwd[LV_WARPS], s_rev[LV_WARPS];
  __shared__ uint32_t s_min;
  const uint32_t nt = L.ctl->n_tiles;
  for (uint32_t w = blockIdx.x; w < 3 * nt; w += gridDim.x) {
    const uint32_t axis = w / nt, t = w % nt;
    const LTile tl = L.tile[b][t];
    const LNode nd = L.node[b][tl.node];
    const uint32_t n = min(LV_TILE, nd.count - tl.off);
    const int32_t* A = L.A[b] + (size_t)axis * L.T + nd.start + tl.off;
    if (threadIdx.x == 0) s_min = 0xffffffffu;
    FBox bx[LV_ITEMS];
#pragma unroll
    for (int j = 0; j < LV_ITEMS; j++) {
      const uint32_t i = threadIdx.x * LV_ITEMS + j;
      bx[j] = i < n ? load_fbox(L.fbox, (uint32_t)A[i]) : fbox_empty();
    }
    float f[LV_ITEMS], g[LV_ITEMS];
    const size_t o = (size_t)axis * L.max_tiles + t;
    tile_scan<false>(bx, L.carry[0][o], s_fwd, [&](int j, const FBox& r) { f[j] = fbox_sa(r); });
    tile_scan<true>(bx, L.carry[1][o], s_rev, [&](int j, const FBox& r) { g[j] = fbox_sa(r); });
    const float inv = 1.0f / fbox_sa(L.nbox[tl.node]);
    uint32_t best = 0xffffffffu;
    float* out = L.cost + (size_t)axis * L.T + nd.start + tl.off;
#pragma unroll
    for (int j = 0; j < LV_ITEMS; j++) {
      const uint32_t i = threadIdx.x * LV_ITEMS + j;
      if (i < n) {
        const uint32_t p = tl.off + i;
        const float c = 0.5f + (f[j] * (float)(p + 1) + g[j] * (float)(nd.count - 1 - p)) * inv;
        out[i] = c;
        best = min(best, __float_as_uint(c));
      }
    }
    best = __reduce_min_sync(0xffffffffu, best);
    if ((threadIdx.x & 31) == 0) atomicMin(&s_min, best);
    __syncthreads();
    if (threadIdx.x == 0) {
      L.tmin[o] = s_min;
      atomicMin(L.nmin + 3 * tl.node + axis, s_min);
    }
    __syncthreads();
  }
}

// Exact boxes of the tiles of every (node, axis) that holds a cost near the node's smallest.
__global__ void __launch_bounds__(LV_THREADS) k_lv_exact_reduce(Level L, int b) {
  __shared__ KBox s_box[LV_WARPS];
  const uint32_t nt = L.ctl->n_tiles;
  for (uint32_t w = blockIdx.x; w < 3 * nt; w += gridDim.x) {
    const uint32_t axis = w / nt, t = w % nt;
    const LTile tl = L.tile[b][t];
    const LNode nd = L.node[b][tl.node];
    if (beyond(L.nmin[3 * tl.node + axis], lv_limit(L, tl.node, nd.count))) continue;
    const uint32_t n = min(LV_TILE, nd.count - tl.off);
    const int32_t* A = L.A[b] + (size_t)axis * L.T + nd.start + tl.off;
    KBox bx = kbox_empty();
    for (uint32_t i = threadIdx.x; i < n; i += LV_THREADS) kbox_add(bx, load_kbox(L.kbox + (uint32_t)A[i]));
    kbox_warp(bx);
    if ((threadIdx.x & 31) == 0) s_box[threadIdx.x >> 5] = bx;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int k = 1; k < LV_WARPS; k++) kbox_add(bx, s_box[k]);
      L.etbox[(size_t)axis * L.max_tiles + t] = bx;
    }
    __syncthreads();
  }
}
template <bool REV>
__device__ __forceinline__ KBox lv_exact_carry(const KBox* in, KBox* out, uint32_t n, int lane) {
  KBox run = kbox_empty();
  for (uint32_t base = 0; base < n; base += 32) {
    const uint32_t i = base + (uint32_t)lane;
    KBox v = i < n ? in[REV ? n - 1 - i : i] : kbox_empty();
    for (int o = 1; o < 32; o <<= 1) {
      const KBox u = kbox_shfl_from<false>(v, o);
      if (lane >= o) kbox_add(v, u);
    }
    KBox ex = kbox_shfl_from<false>(v, 1);
    if (lane == 0) ex = kbox_empty();
    kbox_add(ex, run);
    if (i < n) out[REV ? n - 1 - i : i] = ex;
    KBox last;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      last.mn[a] = __shfl_sync(0xffffffffu, v.mn[a], 31);
      last.mx[a] = __shfl_sync(0xffffffffu, v.mx[a], 31);
    }
    kbox_add(run, last);
  }
  return run;
}
__global__ void __launch_bounds__(LV_THREADS) k_lv_exact_carry(Level L, int b) {
  const int lane = threadIdx.x & 31;
  const uint32_t items = 3 * L.ctl->n_nodes;
  for (uint32_t w = (blockIdx.x * LV_THREADS + threadIdx.x) >> 5; w < items; w += (gridDim.x * LV_THREADS) >> 5) {
    const uint32_t k = w / 3, axis = w % 3;
    const LNode nd = L.node[b][k];
    const float limit = lv_limit(L, k, nd.count);
    if (beyond(L.nmin[w], limit)) continue;
    const size_t o = (size_t)axis * L.max_tiles + nd.tile0;
    const KBox all = lv_exact_carry<false>(L.etbox + o, L.ecarry[0] + o, nd.ntiles, lane);
    lv_exact_carry<true>(L.etbox + o, L.ecarry[1] + o, nd.ntiles, lane);
    bool first = true;  // the node's box: the same from every axis, written by the first near one
    for (uint32_t a = 0; a < axis; a++) first = first && beyond(L.nmin[3 * k + a], limit);
    if (lane == 0 && first) L.nexact[k] = all;
  }
}

// The double costs of the positions near the node's smallest; per tile the
// first smallest of them.
template <bool REV, class F>
__device__ __forceinline__ void tile_scan_exact(const KBox (&bx)[LV_ITEMS], const KBox& carry, KBox* s_warp, F f) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  KBox inc = bx[0];
#pragma unroll
  for (int j = 1; j < LV_ITEMS; j++) kbox_add(inc, bx[j]);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const KBox u = kbox_shfl_from<REV>(inc, o);
    if (REV ? lane + o < 32 : lane >= o) kbox_add(inc, u);
  }
  if (lane == (REV ? 0 : 31)) s_warp[warp] = inc;
  __syncthreads();
  KBox run = kbox_shfl_from<REV>(inc, 1);
  if (lane == (REV ? 31 : 0)) run = kbox_empty();
  kbox_add(run, carry);
  for (int k = 0; k < LV_WARPS; k++)
    if (REV ? k > warp : k < warp) kbox_add(run, s_warp[k]);
#pragma unroll
  for (int q = 0; q < LV_ITEMS; q++) {
    const int j = REV ? LV_ITEMS - 1 - q : q;
    kbox_add(run, bx[j]);
    f(j, run);
  }
}
__device__ __forceinline__ bool better(double c, uint32_t key, double bc, uint32_t bkey) {
  return c < bc || (c == bc && key < bkey);
}
__global__ void __launch_bounds__(LV_THREADS) k_lv_exact(Level L, int b) {
  __shared__ KBox s_fwd[LV_WARPS], s_rev[LV_WARPS];
  __shared__ double s_cost[LV_WARPS];
  __shared__ uint32_t s_key[LV_WARPS];
  const uint32_t nt = L.ctl->n_tiles;
  const double inf = __longlong_as_double(0x7ff0000000000000ll);
  for (uint32_t w = blockIdx.x; w < 3 * nt; w += gridDim.x) {
    const uint32_t axis = w / nt, t = w % nt;
    const LTile tl = L.tile[b][t];
    const LNode nd = L.node[b][tl.node];
    const float limit = lv_limit(L, tl.node, nd.count);
    const size_t o = (size_t)axis * L.max_tiles + t;
    if (beyond(L.tmin[o], limit)) {
      if (threadIdx.x == 0) L.best[o] = Best{inf, ~0u, 0u};
      continue;
    }
    const uint32_t n = min(LV_TILE, nd.count - tl.off);
    const int32_t* A = L.A[b] + (size_t)axis * L.T + nd.start + tl.off;
    const float* approx = L.cost + (size_t)axis * L.T + nd.start + tl.off;
    KBox bx[LV_ITEMS];
    bool near_[LV_ITEMS];
#pragma unroll
    for (int j = 0; j < LV_ITEMS; j++) {
      const uint32_t i = threadIdx.x * LV_ITEMS + j;
      bx[j] = i < n ? load_kbox(L.kbox + (uint32_t)A[i]) : kbox_empty();
      near_[j] = i < n && !(approx[i] > limit);
    }
    double f[LV_ITEMS], g[LV_ITEMS];
    tile_scan_exact<false>(bx, L.ecarry[0][o], s_fwd, [&](int j, const KBox& r) { if (near_[j]) f[j] = kbox_sa(r); });
    tile_scan_exact<true>(bx, L.ecarry[1][o], s_rev, [&](int j, const KBox& r) { if (near_[j]) g[j] = kbox_sa(r); });
    double bc = inf;
    uint32_t bkey = ~0u;
    const double psa = kbox_sa(L.nexact[tl.node]);
#pragma unroll
    for (int j = 0; j < LV_ITEMS; j++) {
      if (!near_[j]) continue;
      const uint32_t p = tl.off + threadIdx.x * LV_ITEMS + j;
      const double c = sweep_cost(f[j], g[j], psa, p, nd.count);
      if (c < bc) { bc = c; bkey = axis * nd.count + p; }
    }
    for (int s = 16; s; s >>= 1) {
      const double oc = __shfl_xor_sync(0xffffffffu, bc, s);
      const uint32_t ok = __shfl_xor_sync(0xffffffffu, bkey, s);
      if (better(oc, ok, bc, bkey)) { bc = oc; bkey = ok; }
    }
    if ((threadIdx.x & 31) == 0) { s_cost[threadIdx.x >> 5] = bc; s_key[threadIdx.x >> 5] = bkey; }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int k = 1; k < LV_WARPS; k++)
        if (better(s_cost[k], s_key[k], bc, bkey)) { bc = s_cost[k]; bkey = s_key[k]; }
      L.best[o] = Best{bc, bkey, 0u};
    }
    __syncthreads();
  }
}

// One warp per node: the first smallest cost.  A node without a finite cost (the
// reference throws there) and a leaf (cost > n, bvh.js:127-143) of more than
// 127 triangles, which the packed leaf word cannot hold, fail the build.
__global__ void __launch_bounds__(LV_THREADS) k_lv_decide(Level L, int b) {
  const int lane = threadIdx.x & 31;
  const uint32_t m = L.ctl->n_nodes;
  const double inf = __longlong_as_double(0x7ff0000000000000ll);
  for (uint32_t k = (blockIdx.x * LV_THREADS + threadIdx.x) >> 5; k < m; k += (gridDim.x * LV_THREADS) >> 5) {
    const LNode nd = L.node[b][k];
    double bc = inf;
    uint32_t bkey = ~0u;
    for (uint32_t i = lane; i < 3 * nd.ntiles; i += 32) {
      const Best r = L.best[(size_t)(i / nd.ntiles) * L.max_tiles + nd.tile0 + i % nd.ntiles];
      if (better(r.cost, r.key, bc, bkey)) { bc = r.cost; bkey = r.key; }
    }
    for (int s = 16; s; s >>= 1) {
      const double oc = __shfl_xor_sync(0xffffffffu, bc, s);
      const uint32_t ok = __shfl_xor_sync(0xffffffffu, bkey, s);
      if (better(oc, ok, bc, bkey)) { bc = oc; bkey = ok; }
    }
    if (lane == 0) {
      uint32_t axis = 0, nl = nd.count / 2;
      const uint32_t idx = bkey == ~0u ? nd.count : bkey % nd.count;
      if (bkey == ~0u || bc > (double)nd.count || idx + 1 >= nd.count) {
        atomicOr(&L.ctl->err, ERR_BVH);
      } else {
        axis = bkey / nd.count;
        nl = idx + 1;
      }
      L.split[k] = axis;
      L.nleft[k] = nl;
      const uint32_t at = L.ctl->n_big + k;
      L.big_start[at] = nd.start;
      L.big_box[at] = L.nexact[k];
    }
  }
}

// #splitNode (bvh.js:80-107): mark the left refs along the split axis ...
__global__ void __launch_bounds__(LV_THREADS) k_lv_flag(Level L, int b) {
  const uint32_t nt = L.ctl->n_tiles;
  for (uint32_t t = blockIdx.x; t < nt; t += gridDim.x) {
    const LTile tl = L.tile[b][t];
    const LNode nd = L.node[b][tl.node];
    const uint32_t n = min(LV_TILE, nd.count - tl.off), nl = L.nleft[tl.node];
    const int32_t* A = L.A[b] + (size_t)L.split[tl.node] * L.T + nd.start + tl.off;
    for (uint32_t i = threadIdx.x; i < n; i += LV_THREADS) L.left[A[i]] = tl.off + i < nl ? 1 : 0;
  }
}
// ... count them per tile of the other two lists ...
__global__ void __launch_bounds__(LV_THREADS) k_lv_count(Level L, int b) {
  __shared__ uint32_t s_n;
  const uint32_t nt = L.ctl->n_tiles;
  for (uint32_t w = blockIdx.x; w < 3 * nt; w += gridDim.x) {
    const uint32_t axis = w / nt, t = w % nt;
    const LTile tl = L.tile[b][t];
    if (L.split[tl.node] == axis) continue;
    const LNode nd = L.node[b][tl.node];
    const uint32_t n = min(LV_TILE, nd.count - tl.off);
    const int32_t* A = L.A[b] + (size_t)axis * L.T + nd.start + tl.off;
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    uint32_t c = 0;
    for (uint32_t i = threadIdx.x; i < n; i += LV_THREADS) c += L.left[A[i]];
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(&s_n, c);
    __syncthreads();
    if (threadIdx.x == 0) L.tcount[(size_t)axis * L.max_tiles + t] = s_n;
    __syncthreads();
  }
}
__global__ void __launch_bounds__(LV_THREADS) k_lv_offsets(Level L, int b) {
  const int lane = threadIdx.x & 31;
  const uint32_t items = 3 * L.ctl->n_nodes;
  for (uint32_t w = (blockIdx.x * LV_THREADS + threadIdx.x) >> 5; w < items; w += (gridDim.x * LV_THREADS) >> 5) {
    const uint32_t k = w / 3, axis = w % 3;
    if (L.split[k] == axis) continue;
    const LNode nd = L.node[b][k];
    uint32_t* c = L.tcount + (size_t)axis * L.max_tiles + nd.tile0;
    uint32_t run = 0;
    for (uint32_t base = 0; base < nd.ntiles; base += 32) {
      const uint32_t i = base + (uint32_t)lane;
      const uint32_t v = i < nd.ntiles ? c[i] : 0u;
      uint32_t inc = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
      }
      if (i < nd.ntiles) c[i] = run + inc - v;
      run += __shfl_sync(0xffffffffu, inc, 31);
    }
  }
}
// ... and partition every list stably into the children's ranges.
__global__ void __launch_bounds__(LV_THREADS) k_lv_scatter(Level L, int b) {
  __shared__ uint32_t s_warp[LV_WARPS + 1][2];
  const uint32_t nt = L.ctl->n_tiles;
  for (uint32_t w = blockIdx.x; w < 3 * nt; w += gridDim.x) {
    const uint32_t axis = w / nt, t = w % nt;
    const LTile tl = L.tile[b][t];
    const LNode nd = L.node[b][tl.node];
    const uint32_t n = min(LV_TILE, nd.count - tl.off);
    const size_t list = (size_t)axis * L.T + nd.start;
    const int32_t* A = L.A[b] + list + tl.off;
    int32_t* out = L.A[b ^ 1] + list;
    if (L.split[tl.node] == axis) {  // already in order
      for (uint32_t i = threadIdx.x; i < n; i += LV_THREADS) out[tl.off + i] = A[i];
      continue;
    }
    int32_t id[LV_ITEMS];
    uint32_t fl = 0, c = 0;
#pragma unroll
    for (int j = 0; j < LV_ITEMS; j++) {
      const uint32_t i = threadIdx.x * LV_ITEMS + j;
      id[j] = i < n ? A[i] : 0;
      const uint32_t f = i < n ? L.left[id[j]] : 0u;
      fl |= f << j;
      c += f;
    }
    uint32_t ea, eb, ta, tb;
    block_scan2<LV_WARPS>(c, 0u, ea, eb, ta, tb, s_warp);
    uint32_t before = L.tcount[(size_t)axis * L.max_tiles + t] + ea;  // left triangles before this position
    const uint32_t nl = L.nleft[tl.node];
#pragma unroll
    for (int j = 0; j < LV_ITEMS; j++) {
      const uint32_t i = threadIdx.x * LV_ITEMS + j;
      if (i >= n) break;
      const bool f = (fl >> j) & 1u;
      const uint32_t to = f ? before : nl + (tl.off + i - before);
      if (to < nd.count) out[to] = id[j];
      else atomicOr(&L.ctl->err, ERR_BVH);
      before += f;
    }
    __syncthreads();
  }
}

// One block: the next level's nodes and tiles in order of position, and the
// children small enough for phase 2.
constexpr int NEXT_THREADS = 1024;
__global__ void __launch_bounds__(NEXT_THREADS) k_lv_next(Level L, int b, uint32_t level) {
  __shared__ uint32_t s_warp[NEXT_THREADS / 32 + 1][2];
  const uint32_t m = L.ctl->n_nodes;
  uint32_t nodes = 0, tiles = 0;
  for (uint32_t base = 0; base < m; base += NEXT_THREADS) {
    const uint32_t k = base + threadIdx.x;
    LNode ch[2];
    uint32_t cn = 0, ct = 0;
    if (k < m) {
      const LNode nd = L.node[b][k];
      const uint32_t nl = L.nleft[k];
      ch[0] = LNode{nd.start, nl, 0u, 0u};
      ch[1] = LNode{nd.start + nl, nd.count - nl, 0u, 0u};
      for (int s = 0; s < 2; s++) {
        if (ch[s].count > SUB) {
          ch[s].ntiles = (ch[s].count + LV_TILE - 1) / LV_TILE;
          cn++;
          ct += ch[s].ntiles;
        } else {
          L.small[atomicAdd(&L.ctl->n_small, 1u)] = SmallTask{ch[s].start, ch[s].count, level + 1, (uint32_t)(b ^ 1)};
        }
      }
    }
    uint32_t en, et, tn, tt;
    block_scan2<NEXT_THREADS / 32>(cn, ct, en, et, tn, tt, s_warp);
    uint32_t at = nodes + en, t0 = tiles + et;
    if (k < m)
      for (int s = 0; s < 2; s++)
        if (ch[s].ntiles) {
          ch[s].tile0 = t0;
          L.node[b ^ 1][at++] = ch[s];
          t0 += ch[s].ntiles;
        }
    nodes += tn;
    tiles += tt;
    __syncthreads();
  }
  __threadfence_block();
  __syncthreads();
  for (uint32_t t = threadIdx.x; t < tiles; t += NEXT_THREADS) {
    uint32_t lo = 0, hi = nodes - 1;  // the last node whose first tile is not after t
    while (lo < hi) {
      const uint32_t mid = (lo + hi + 1) >> 1;
      if (L.node[b ^ 1][mid].tile0 <= t) lo = mid; else hi = mid - 1;
    }
    L.tile[b ^ 1][t] = LTile{lo, (t - L.node[b ^ 1][lo].tile0) * LV_TILE};
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const uint32_t big = L.ctl->n_big + m;
    L.ctl->n_big = big;
    L.big_off[level + 1] = big;
    L.ctl->n_nodes = nodes;
    L.ctl->n_tiles = tiles;
  }
}

// =====================================================================
// Phase 2: one block builds the whole subtree of a node of at most SUB
// triangles in shared memory, level by level over all nodes of the level at
// once: segmented scans of the rounded boxes along the three lists, binary32
// costs, the near ones again in double, a stable partition.
// Bound by barrier and instruction-fetch latency (29% of issue slots with the six
// scans of a level inlined one after the other, so the three lists share one copy
// of their two scans and keep their costs in shared memory); 256 threads of two
// positions each, 4 blocks (51 KB, 64 registers) on an SM.  Whole build of
// 1,310,730 triangles: six scans inlined, 128 threads 8.02 ms; one copy, 128
// threads 7.77 (96 registers: 4 blocks), 256 threads 7.53 (3 blocks 7.70), 512
// threads of one position 8.45.
// =====================================================================
constexpr int ST_THREADS = 256;
constexpr int ST_BLOCKS = 4;
constexpr int ST_PER = (int)SUB / ST_THREADS;
constexpr int ST_WARPS = ST_THREADS / 32;
constexpr uint16_t NO_NODE = 0xffff;

struct SubNode {       // a node of a subtree, in the subtree's BFS order
  uint32_t level, rank;  // level below the subtree's root, rank in it
  uint32_t leaf;         // triangles of a leaf, 0: inner
  uint32_t order;        // inner: rank among the level's inner nodes; leaf: triangles of the level's leaves before it
  uint32_t pos;          // leaf: first position of its triangles (leaf_ids)
};
struct Subtrees {
  Ctl* ctl;
  const KBox* kbox;
  const int32_t* A[2];
  uint32_t T;
  const SmallTask* task;  // in order of position
  SubNode* node;          // [2 T], subtree s from 2 * start
  KBox* box;              // the same index
  uint32_t* leaf_ids;     // [T]
  uint32_t* lv_inner;     // [T], subtree s from its start: inner nodes per level
  uint32_t* lv_leaf;      // triangles in leaves per level
  uint32_t* depth;        // per subtree
  uint32_t* count;        // per subtree: nodes
  uint16_t* local;        // [T] triangle -> its number in the subtree
};

struct StShared {
  uint32_t fb[6][SUB];
  uint32_t gid[SUB];
  uint16_t lst[2][3][SUB];
  uint16_t seg[2][SUB];
  uint16_t nst[2][SUB], ncn[2][SUB];
  uint32_t nmin[SUB];    // smallest cost (bits)
  float bound[SUB];      // the node's E
  float inv[SUB];        // 1 / its area
  uint32_t first[SUB];   // first near cost: axis * count + index
  uint32_t dec[SUB];     // axis << 30 | leaf << 29 | nleft
  uint16_t irank[SUB];
  uint16_t todo[SUB];    // nodes that need double costs
  uint32_t pre[SUB];     // left triangles before a position: 10 bits per list
  uint32_t near_[3][SUB / 32];
  uint8_t left[SUB];
  float cost[3][SUB];
  FBox wbox[2][ST_WARPS];
  uint32_t wflag[2][ST_WARPS];
  uint32_t warp[ST_WARPS + 1][2];
  KBox kwarp[ST_WARPS];
  uint32_t lvbase[SUB + 1];
  uint32_t n_todo;
};

// Segmented running areas along one list, forwards or backwards (each direction
// has its shared words); emit(j, box, area) for the running box at position j.
template <bool REV, class Emit>
__device__ __forceinline__ void seg_areas(StShared& S, const uint16_t* lst, const uint16_t (&sg)[ST_PER],
                                          uint32_t edge, float (&area)[ST_PER], Emit emit) {
  constexpr int SLOT = REV ? 1 : 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  FBox bx[ST_PER];
  FBox inc = fbox_empty();
  bool fl = false;
#pragma unroll
  for (int q = 0; q < ST_PER; q++) {
    const int j = REV ? ST_PER - 1 - q : q;
    bx[j] = fbox_empty();
    if (sg[j] != NO_NODE) {
      const uint32_t id = lst[threadIdx.x * ST_PER + j];
#pragma unroll
      for (int a = 0; a < 3; a++) { bx[j].mn[a] = S.fb[a][id]; bx[j].mx[a] = S.fb[3 + a][id]; }
    }
    if ((edge >> j) & 1u) { inc = bx[j]; fl = true; }
    else fbox_add(inc, bx[j]);
  }
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const FBox u = fbox_shfl_from<REV>(inc, o);
    const bool uf = REV ? __shfl_down_sync(0xffffffffu, fl, o) : __shfl_up_sync(0xffffffffu, fl, o);
    if (REV ? lane + o < 32 : lane >= o) {
      if (!fl) fbox_add(inc, u);
      fl = fl || uf;
    }
  }
  if (lane == (REV ? 0 : 31)) { S.wbox[SLOT][warp] = inc; S.wflag[SLOT][warp] = fl; }
  __syncthreads();
  FBox run = fbox_empty();
  for (int q = 0; q < ST_WARPS; q++) {  // the warps before this one in scan order
    const int k = REV ? ST_WARPS - 1 - q : q;
    if (REV ? k > warp : k < warp) {
      if (S.wflag[SLOT][k]) run = S.wbox[SLOT][k];
      else fbox_add(run, S.wbox[SLOT][k]);
    }
  }
  const FBox lb = fbox_shfl_from<REV>(inc, 1);
  const bool lf = REV ? __shfl_down_sync(0xffffffffu, fl, 1) : __shfl_up_sync(0xffffffffu, fl, 1);
  if (lane != (REV ? 31 : 0)) {
    if (lf) run = lb;
    else fbox_add(run, lb);
  }
#pragma unroll
  for (int q = 0; q < ST_PER; q++) {
    const int j = REV ? ST_PER - 1 - q : q;
    if ((edge >> j) & 1u) run = bx[j];
    else fbox_add(run, bx[j]);
    area[j] = fbox_sa(run);
    emit(j, run, area[j]);
  }
}

// Exact cost of (axis, i) of the node at [st, st + n), by one warp.
__device__ __forceinline__ double exact_cost(const StShared& S, const KBox* kbox, const uint16_t* lst, uint32_t st,
                                             uint32_t n, uint32_t i, double psa, KBox* whole) {
  const uint32_t lane = threadIdx.x & 31;
  KBox f = kbox_empty(), g = kbox_empty();
  for (uint32_t j = lane; j < n; j += 32) {
    const KBox k = load_kbox(kbox + S.gid[lst[st + j]]);
    if (j <= i) kbox_add(f, k);
    if (j >= i) kbox_add(g, k);
  }
  kbox_warp(f);
  kbox_warp(g);
  if (whole) {
    *whole = f;
    kbox_add(*whole, g);
    psa = kbox_sa(*whole);
  }
  return sweep_cost(kbox_sa(f), kbox_sa(g), psa, i, n);
}

__global__ void __launch_bounds__(ST_THREADS, ST_BLOCKS) k_subtree(Subtrees W) {
  extern __shared__ __align__(16) unsigned char st_raw[];
  StShared& S = *reinterpret_cast<StShared*>(st_raw);
  if (W.ctl->err & ERR_LOOKBACK) return;  // the tasks were not placed; this kernel sets other bits only
  const SmallTask task = W.task[blockIdx.x];
  const uint32_t n0 = task.count, start = task.start;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int32_t* A = W.A[task.buf];
  // triangles numbered by the first list; rounded boxes in the subtree's frame
  KBox all = kbox_empty();
  for (uint32_t i = tid; i < n0; i += ST_THREADS) {
    const uint32_t g = (uint32_t)A[start + i];
    S.gid[i] = g;
    W.local[g] = (uint16_t)i;
    S.lst[0][0][i] = (uint16_t)i;
    kbox_add(all, load_kbox(W.kbox + g));
  }
  kbox_warp(all);
  if (lane == 0) S.kwarp[warp] = all;
  __threadfence_block();
  __syncthreads();
  all = S.kwarp[0];
  for (int k = 1; k < ST_WARPS; k++) kbox_add(all, S.kwarp[k]);
  const Frame fr = frame_of(all);
  for (uint32_t i = tid; i < SUB; i += ST_THREADS) {
    S.seg[0][i] = i < n0 ? 0 : NO_NODE;
    if (i >= n0) continue;
    const KBox k = load_kbox(W.kbox + S.gid[i]);
#pragma unroll
    for (int a = 0; a < 3; a++) {
      S.fb[a][i] = rounded(val_of(k.mn[a]), fr.lo[a], fr.scale);
      S.fb[3 + a][i] = rounded(val_of(k.mx[a]), fr.lo[a], fr.scale);
    }
    S.lst[0][1][i] = __ldcg(W.local + A[(size_t)W.T + start + i]);
    S.lst[0][2][i] = __ldcg(W.local + A[2 * (size_t)W.T + start + i]);
  }
  if (tid == 0) {
    S.nst[0][0] = 0;
    S.ncn[0][0] = (uint16_t)n0;
    S.lvbase[0] = 0;
  }
  uint32_t m = 1, base = 0, level = 0;
  int b = 0;
  uint32_t inner_total = 0;
  __syncthreads();
  while (m) {
    for (uint32_t k = tid; k < m; k += ST_THREADS) { S.nmin[k] = 0xffffffffu; S.first[k] = 0xffffffffu; }
    if (tid < 3 * (int)SUB / 32) (&S.near_[0][0])[tid] = 0u;
    if (tid == 0) S.n_todo = 0;
    // costs
    uint16_t sg[ST_PER];
    uint32_t head = 0, tail = 0, st[ST_PER], cn[ST_PER];
#pragma unroll
    for (int j = 0; j < ST_PER; j++) {
      const uint32_t p = tid * ST_PER + j;
      sg[j] = S.seg[b][p];
      st[j] = cn[j] = 0;
      if (sg[j] == NO_NODE) {
        head |= 1u << j;
        tail |= 1u << j;
      } else {
        st[j] = S.nst[b][sg[j]];
        cn[j] = S.ncn[b][sg[j]];
        if (p == st[j]) head |= 1u << j;
        if (p == st[j] + cn[j] - 1) tail |= 1u << j;
      }
    }
    // one copy of the scans for the three lists
    uint32_t c3[ST_PER];
#pragma unroll
    for (int j = 0; j < ST_PER; j++) c3[j] = 0xffffffffu;
#pragma unroll 1
    for (int a = 0; a < 3; a++) {
      const uint16_t* lst = S.lst[b][a];
      float f[ST_PER], g[ST_PER];
      seg_areas<false>(S, lst, sg, head, f, [&](int j, const FBox& run, float area) {
        if (a == 0 && sg[j] != NO_NODE && ((tail >> j) & 1u)) {  // the node's box
          S.bound[sg[j]] = cost_bound(run, cn[j], fr.ok);
          S.inv[sg[j]] = 1.0f / area;
        }
      });
      seg_areas<true>(S, lst, sg, tail, g, [](int, const FBox&, float) {});
#pragma unroll
      for (int j = 0; j < ST_PER; j++) {
        if (sg[j] == NO_NODE) continue;
        const uint32_t i = tid * ST_PER + j - st[j];
        const float cost = 0.5f + (f[j] * (float)(i + 1) + g[j] * (float)(cn[j] - 1 - i)) * S.inv[sg[j]];
        S.cost[a][tid * ST_PER + j] = cost;
        c3[j] = min(c3[j], __float_as_uint(cost));
      }
    }
    // a warp inside one node (its range is contiguous) combines its costs before the shared atomic
    const int s_first = sg[0], s_last = sg[ST_PER - 1], s_lane0 = __shfl_sync(0xffffffffu, s_first, 0);
    const bool one = __all_sync(0xffffffffu, s_first != NO_NODE && s_first == s_last && s_first == s_lane0);
    uint32_t low = 0xffffffffu;
#pragma unroll
    for (int j = 0; j < ST_PER; j++) {
      if (sg[j] == NO_NODE) continue;
      if (one) low = min(low, c3[j]);
      else atomicMin(&S.nmin[sg[j]], c3[j]);
    }
    if (one) {
      low = __reduce_min_sync(0xffffffffu, low);
      if (lane == 0) atomicMin(&S.nmin[sg[0]], low);
    }
    __syncthreads();
    // positions near the smallest
#pragma unroll
    for (int j = 0; j < ST_PER; j++) {
      if (sg[j] == NO_NODE || cn[j] == 1) continue;
      const uint32_t p = tid * ST_PER + j;
      const float limit = __uint_as_float(S.nmin[sg[j]]) + 2.0f * S.bound[sg[j]];
#pragma unroll
      for (int a = 0; a < 3; a++)
        if (!(S.cost[a][p] > limit)) {
          atomicOr(&S.near_[a][p >> 5], 1u << (p & 31u));
          atomicMin(&S.first[sg[j]], a * cn[j] + (p - st[j]));
        }
    }
    __syncthreads();
    // nodes the binary32 costs decide
    for (uint32_t k = tid; k < m; k += ST_THREADS) {
      const uint32_t n = S.ncn[b][k], s0 = S.nst[b][k];
      const float E = S.bound[k];
      if (n == 1 && E < 1e30f) {  // 0.5 + 1 > 1: a leaf, in any list's order
        S.dec[k] = (1u << 29) | 1u;
        continue;
      }
      bool sure = E < 1e30f;
      if (sure) {
        const float low32 = __uint_as_float(S.nmin[k]);
        sure = low32 - E > (float)n || low32 + E < (float)n;
      }
      uint32_t cands = 0;
      if (sure) {
        // near positions, those of a list in the same order as an earlier one left out: their costs are the same
        for (uint32_t a = 0; a < 3 && cands < 2; a++) {
          if (n <= 8) {
            bool same = false;
            for (uint32_t e = 0; e < a && !same; e++) {
              same = true;
              for (uint32_t i = 0; i < n && same; i++) same = S.lst[b][a][s0 + i] == S.lst[b][e][s0 + i];
            }
            if (same) continue;
          }
          for (uint32_t wd = s0 >> 5; wd <= (s0 + n - 1) >> 5; wd++) {
            uint32_t bits = S.near_[a][wd];
            if (wd == s0 >> 5) bits &= 0xffffffffu << (s0 & 31u);
            if (wd == (s0 + n - 1) >> 5) bits &= 0xffffffffu >> (31u - ((s0 + n - 1) & 31u));
            cands += (uint32_t)__popc(bits);
          }
        }
        sure = cands == 1;
      }
      if (sure) {
        const uint32_t key = S.first[k], axis = key / n, idx = key % n;
        const bool leaf = __uint_as_float(S.nmin[k]) > (float)n;
        S.dec[k] = (axis << 30) | (leaf ? 1u << 29 : 0u) | (idx + 1);
      } else {
        S.todo[atomicAdd(&S.n_todo, 1u)] = (uint16_t)k;
      }
    }
    __syncthreads();
    // the others in double, a warp per node
    for (uint32_t q = warp; q < S.n_todo; q += ST_WARPS) {
      const uint32_t k = S.todo[q], n = S.ncn[b][k], s0 = S.nst[b][k];
      double best = __longlong_as_double(0x7ff0000000000000ll), psa = 0.0;
      uint32_t key = ~0u;
      bool known = false;
      for (uint32_t a = 0; a < 3; a++)
        for (uint32_t wd = s0 >> 5; wd <= (s0 + n - 1) >> 5; wd++) {
          uint32_t bits = n == 1 ? 1u << (s0 & 31u) : S.near_[a][wd];
          if (wd == s0 >> 5) bits &= 0xffffffffu << (s0 & 31u);
          if (wd == (s0 + n - 1) >> 5) bits &= 0xffffffffu >> (31u - ((s0 + n - 1) & 31u));
          while (bits) {
            const uint32_t i = wd * 32u + (uint32_t)__ffs(bits) - 1u - s0;
            bits &= bits - 1u;
            KBox whole;
            const double c = exact_cost(S, W.kbox, S.lst[b][a], s0, n, i, psa, known ? nullptr : &whole);
            if (!known) { psa = kbox_sa(whole); known = true; }
            if (c < best) { best = c; key = a * n + i; }
          }
        }
      if (lane == 0) {
        bool leaf = best > (double)n;
        if (key == ~0u) {  // no finite split cost: the reference throws here
          atomicOr(&W.ctl->err, ERR_BVH);
          leaf = true;
          key = 0;
        }
        if (leaf && n >= 128u) atomicOr(&W.ctl->err, ERR_BVH);  // does not fit the packed leaf word
        if (!leaf && key % n + 1 >= n) { atomicOr(&W.ctl->err, ERR_BVH); leaf = true; }
        S.dec[k] = ((key / n) << 30) | (leaf ? 1u << 29 : 0u) | (key % n + 1);
      }
    }
    __syncthreads();
    // ranks of inner nodes and leaf triangles in the level
    uint32_t inner = 0, leaves = 0;
    for (uint32_t k0 = 0; k0 < m; k0 += ST_THREADS) {
      const uint32_t k = k0 + tid;
      const uint32_t d = k < m ? S.dec[k] : 0u;
      const bool leaf = (d >> 29) & 1u;
      const uint32_t n = k < m ? S.ncn[b][k] : 0u;
      uint32_t ei, el, ti, tl;
      block_scan2<ST_WARPS>(k < m && !leaf ? 1u : 0u, leaf ? n : 0u, ei, el, ti, tl, S.warp);
      if (k < m) {
        S.irank[k] = (uint16_t)(inner + ei);
        if (leaf && n >= 128u) atomicOr(&W.ctl->err, ERR_BVH);
        W.node[2 * (size_t)start + base + k] =
            SubNode{level, k, leaf ? n : 0u, leaf ? leaves + el : inner + ei, start + S.nst[b][k]};
      }
      inner += ti;
      leaves += tl;
      __syncthreads();
    }
    // left refs; leaf triangles in the order of the best axis
#pragma unroll
    for (int j = 0; j < ST_PER; j++) {
      if (sg[j] == NO_NODE) continue;
      const uint32_t p = tid * ST_PER + j, d = S.dec[sg[j]];
      const uint32_t id = S.lst[b][d >> 30][p];
      if ((d >> 29) & 1u) W.leaf_ids[start + p] = S.gid[id];
      else S.left[id] = (p - st[j]) < (d & 0x1fffffffu) ? 1 : 0;
    }
    __syncthreads();
    // stable partition of the three lists
    uint32_t fl[3] = {0u, 0u, 0u}, packed = 0;
#pragma unroll
    for (int j = 0; j < ST_PER; j++) {
      if (sg[j] == NO_NODE || ((S.dec[sg[j]] >> 29) & 1u)) continue;
#pragma unroll
      for (int a = 0; a < 3; a++) {
        const uint32_t l = S.left[S.lst[b][a][tid * ST_PER + j]];
        fl[a] |= l << j;
        packed += l << (10 * a);
      }
    }
    uint32_t ep, dummy, tp, dummy2;
    block_scan2<ST_WARPS>(packed, 0u, ep, dummy, tp, dummy2, S.warp);
    {
      uint32_t run = ep;
#pragma unroll
      for (int j = 0; j < ST_PER; j++) {
        S.pre[tid * ST_PER + j] = run;
#pragma unroll
        for (int a = 0; a < 3; a++) run += ((fl[a] >> j) & 1u) << (10 * a);
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ST_PER; j++) {
      const uint32_t p = tid * ST_PER + j;
      const uint32_t d = sg[j] != NO_NODE ? S.dec[sg[j]] : 1u << 29;
      if ((d >> 29) & 1u) {
        S.seg[b ^ 1][p] = NO_NODE;
        continue;
      }
      const uint32_t nl = d & 0x1fffffffu, i = p - st[j];
      const uint32_t mine = S.pre[p], first = S.pre[st[j]];
      const uint16_t r2 = (uint16_t)(2 * S.irank[sg[j]]);
#pragma unroll
      for (int a = 0; a < 3; a++) {
        const uint32_t x = ((mine >> (10 * a)) & 1023u) - ((first >> (10 * a)) & 1023u);
        const bool l = (fl[a] >> j) & 1u;
        const uint32_t to = st[j] + (l ? x : nl + (i - x));
        S.lst[b ^ 1][a][to] = S.lst[b][a][p];
        if (a == 0) S.seg[b ^ 1][to] = r2 + (l ? 0 : 1);
      }
    }
    for (uint32_t k = tid; k < m; k += ST_THREADS) {
      const uint32_t d = S.dec[k];
      if ((d >> 29) & 1u) continue;
      const uint32_t r = S.irank[k], nl = d & 0x1fffffffu;
      S.nst[b ^ 1][2 * r] = S.nst[b][k];
      S.ncn[b ^ 1][2 * r] = (uint16_t)nl;
      S.nst[b ^ 1][2 * r + 1] = (uint16_t)(S.nst[b][k] + nl);
      S.ncn[b ^ 1][2 * r + 1] = (uint16_t)(S.ncn[b][k] - nl);
    }
    if (tid == 0) {
      W.lv_inner[start + level] = inner;
      W.lv_leaf[start + level] = leaves;
      S.lvbase[level + 1] = base + m;
    }
    inner_total += inner;
    base += m;
    m = 2 * inner;
    level++;
    b ^= 1;
    __syncthreads();
  }
  // exact node boxes from the leaves up
  const SubNode* nodes = W.node + 2 * (size_t)start;
  KBox* boxes = W.box + 2 * (size_t)start;
  for (uint32_t l = level; l-- > 0;) {
    const uint32_t e = S.lvbase[l + 1];
    for (uint32_t k = S.lvbase[l] + tid; k < e; k += ST_THREADS) {
      const SubNode nd = nodes[k];
      KBox bx;
      if (nd.leaf) {
        bx = load_kbox(W.kbox + W.leaf_ids[nd.pos]);
        for (uint32_t i = 1; i < nd.leaf; i++) kbox_add(bx, load_kbox(W.kbox + W.leaf_ids[nd.pos + i]));
      } else {
        bx = boxes[e + 2 * nd.order];
        kbox_add(bx, boxes[e + 2 * nd.order + 1]);
      }
      boxes[k] = bx;
    }
    __threadfence_block();
    __syncthreads();
  }
  if (tid == 0) {
    W.depth[blockIdx.x] = level;
    W.count[blockIdx.x] = base;
    atomicAdd(&W.ctl->inner, inner_total);
    atomicMax(&W.ctl->levels, task.level + level);
  }
}

// ---- subtrees in order of position --------------------------------------------------
__global__ void k_mark_tasks(const SmallTask* __restrict__ t, uint32_t n, uint32_t* __restrict__ flag) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) flag[t[i].start] = 1u;
}
__global__ void k_place_tasks(const SmallTask* __restrict__ t, uint32_t n, const uint32_t* __restrict__ rank,
                              SmallTask* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[rank[t[i].start]] = t[i];
}
__global__ void k_one_task(SmallTask* t, uint32_t T, Ctl* c) {
  *t = SmallTask{0u, T, 0u, 0u};
  c->n_small = 1;
}

// ---- BFS order ------------------------------------------------------------------
// Per level (one block): of every subtree, how many nodes, inner nodes and
// leaf triangles lie to its left in that level, large nodes aside.
struct Columns {
  uint32_t *nodes, *inner, *leaf;       // [levels][S]
  uint32_t *level_base, *leaf_off;      // [levels + 1]
  const uint32_t* big_off;              // large nodes before each level, n_lv + 1 entries
  uint32_t n_lv;                        // levels that hold large nodes
  uint32_t S, levels;
};
__device__ __forceinline__ uint32_t large_in(const Columns& C, uint32_t d) {
  return d < C.n_lv ? C.big_off[d + 1] - C.big_off[d] : 0u;
}
constexpr int COL_THREADS = 256;
__global__ void __launch_bounds__(COL_THREADS) k_columns(Subtrees W, Columns C) {
  __shared__ uint32_t s_warp[COL_THREADS / 32 + 1][2];
  const uint32_t d = blockIdx.x;
  uint32_t rn = 0, ri = 0, rl = 0;
  for (uint32_t base = 0; base < C.S; base += COL_THREADS) {
    const uint32_t s = base + threadIdx.x;
    uint32_t nn = 0, ni = 0, nl = 0;
    if (s < C.S) {
      const SmallTask t = W.task[s];
      const uint32_t depth = W.depth[s];
      if (d >= t.level && d - t.level < depth) {
        const uint32_t l = d - t.level;
        nn = l ? 2u * W.lv_inner[t.start + l - 1] : 1u;
        ni = W.lv_inner[t.start + l];
        nl = W.lv_leaf[t.start + l];
      }
    }
    uint32_t en, ei, tn, ti, el, x, tl, y;
    block_scan2<COL_THREADS / 32>(nn, ni, en, ei, tn, ti, s_warp);
    __syncthreads();
    block_scan2<COL_THREADS / 32>(nl, 0u, el, x, tl, y, s_warp);
    if (s < C.S) {
      const size_t o = (size_t)d * C.S + s;
      C.nodes[o] = rn + en;
      C.inner[o] = ri + ei;
      C.leaf[o] = rl + el;
    }
    rn += tn;
    ri += ti;
    rl += tl;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    C.level_base[d + 1] = rn + large_in(C, d);  // this level's nodes; summed below
    C.leaf_off[d + 1] = rl;
  }
}
__global__ void __launch_bounds__(COL_THREADS) k_level_sums(Columns C) {
  __shared__ uint32_t s_warp[COL_THREADS / 32 + 1][2];
  uint32_t rn = 0, rl = 0;
  if (threadIdx.x == 0) C.level_base[0] = C.leaf_off[0] = 0u;
  for (uint32_t base = 0; base < C.levels; base += COL_THREADS) {
    const uint32_t d = base + threadIdx.x;
    const uint32_t a = d < C.levels ? C.level_base[d + 1] : 0u, l = d < C.levels ? C.leaf_off[d + 1] : 0u;
    uint32_t ea, el, ta, tl;
    block_scan2<COL_THREADS / 32>(a, l, ea, el, ta, tl, s_warp);
    if (d < C.levels) {
      C.level_base[d + 1] = rn + ea + a;
      C.leaf_off[d + 1] = rl + el + l;
    }
    rn += ta;
    rl += tl;
    __syncthreads();
  }
}

struct Emit {
  const int4* tri4;
  Norm norm;
  int32_t* nodes5;
  int4* tri4_leaf;
  KBox* node_box;  // doubles on exit
  uint32_t n_nodes, T;
  uint32_t* err;
};
__device__ __forceinline__ void emit_node(const Emit& E, uint32_t bfs, int32_t child, int32_t tris, const KBox& k) {
  if (bfs >= E.n_nodes) { atomicOr(E.err, ERR_BVH); return; }
  double b6[6];
#pragma unroll
  for (int a = 0; a < 3; a++) { b6[a] = val_of(k.mn[a]); b6[3 + a] = val_of(k.mx[a]); }
  int32_t* nd = E.nodes5 + 5 * (size_t)bfs;
  nd[0] = child;
  nd[1] = tris;
#pragma unroll
  for (int a = 0; a < 3; a++) nd[2 + a] = quantize_bounds(E.norm, a, b6[a], b6[3 + a]);
  double2* out = reinterpret_cast<double2*>(E.node_box + bfs);
  out[0] = make_double2(b6[0], b6[1]);
  out[1] = make_double2(b6[2], b6[3]);
  out[2] = make_double2(b6[4], b6[5]);
}
// Large nodes of level d to the left of a position.
__device__ __forceinline__ uint32_t large_before(const Columns& C, const uint32_t* big_start, uint32_t d, uint32_t pos) {
  uint32_t lo = 0, hi = large_in(C, d);
  const uint32_t* s = big_start + (hi ? C.big_off[d] : 0u);
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (s[mid] < pos) lo = mid + 1; else hi = mid;
  }
  return lo;
}
__global__ void __launch_bounds__(128) k_emit_small(Subtrees W, Columns C, Emit E, const uint32_t* __restrict__ big_start) {
  const uint32_t s = blockIdx.x;
  const SmallTask t = W.task[s];
  const uint32_t count = W.count[s];
  for (uint32_t k = threadIdx.x; k < count; k += blockDim.x) {
    const SubNode nd = W.node[2 * (size_t)t.start + k];
    const KBox bx = load_kbox(W.box + 2 * (size_t)t.start + k);
    const uint32_t d = t.level + nd.level;
    const uint32_t big = large_before(C, big_start, d, t.start);
    const size_t col = (size_t)d * C.S + s;
    const uint32_t bfs = C.level_base[d] + big + C.nodes[col] + nd.rank;
    if (nd.leaf) {
      const uint32_t first = C.leaf_off[d] + C.leaf[col] + nd.order;
      if (first >= (1u << 24) || first + nd.leaf > E.T) { atomicOr(E.err, ERR_BVH); continue; }
      for (uint32_t i = 0; i < nd.leaf; i++) E.tri4_leaf[first + i] = E.tri4[W.leaf_ids[nd.pos + i]];
      emit_node(E, bfs, -1, (int32_t)((nd.leaf << 24) | first), bx);  // maskTriIndex (trace_pass.js:166-170)
    } else {
      emit_node(E, bfs, (int32_t)(C.level_base[d + 1] + 2 * (big + C.inner[col] + nd.order)), -1, bx);
    }
  }
}
__global__ void __launch_bounds__(128) k_emit_large(Subtrees W, Columns C, Emit E, const uint32_t* __restrict__ big_start,
                                                    const KBox* __restrict__ big_box, uint32_t n_big) {
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n_big) return;
  uint32_t lo = 0, hi = C.n_lv - 1;  // its level
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1) >> 1;
    if (C.big_off[mid] <= q) lo = mid; else hi = mid - 1;
  }
  const uint32_t d = lo, k = q - C.big_off[d], pos = big_start[q];
  uint32_t a = 0, z = C.S;  // subtrees to its left
  while (a < z) {
    const uint32_t mid = (a + z) >> 1;
    if (W.task[mid].start < pos) a = mid + 1; else z = mid;
  }
  // the subtrees to its left: the prefix at the next one, or the level's sum
  uint32_t left_n, left_i;
  if (a < C.S) {
    left_n = C.nodes[(size_t)d * C.S + a];
    left_i = C.inner[(size_t)d * C.S + a];
  } else {
    left_n = left_i = 0;  // a large node always has subtrees inside it, hence to its right
    atomicOr(E.err, ERR_BVH);
  }
  emit_node(E, C.level_base[d] + k + left_n, (int32_t)(C.level_base[d + 1] + 2 * (k + left_i)), -1, load_kbox(big_box + q));
}

unsigned blocks(uint32_t n, unsigned t = 256) { return (unsigned)((n + t - 1) / t); }

}  // namespace

int build_bvh_sweep(const Scratch& w, const double* pos3, uint32_t n_verts, const int4* tri4, uint32_t T,
                    BvhOut& out, std::string& why) {
  if (T == 0) { why = "no triangles"; return 1; }
  if (T > (1u << 26)) { why = "too many triangles"; return 1; }
  const cudaStream_t s = w.s;
  int dev = 0, sms = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);

  TmpBuf<Ctl> ctl(w, 1);
  k_init<<<1, 1, 0, s>>>(ctl.p);
  uint32_t* err = &ctl.p->err;
  TmpBuf<KBox> kbox(w, T);
  TmpBuf<uint32_t> lists(w, 3 * (size_t)T), lists2(w, 3 * (size_t)T);
  {
    TmpBuf<u64> keys(w, 3 * (size_t)T), keys_tmp(w, 3 * (size_t)T);
    k_tri_boxes<<<blocks(T), TRI_THREADS, 0, s>>>(pos3, tri4, T, kbox.p, keys.p, lists.p, &ctl.p->root);
    check(cudaGetLastError(), "k_tri_boxes");
    radix_sort_pairs_u64(w, reinterpret_cast<uint64_t*>(keys.p), lists.p, reinterpret_cast<uint64_t*>(keys_tmp.p),
                         lists2.p, T, 3, err);
  }
  int32_t* A[2] = {reinterpret_cast<int32_t*>(lists.p), reinterpret_cast<int32_t*>(lists2.p)};

  Ctl host;
  auto read_ctl = [&]() {
    check(cudaMemcpyAsync(&host, ctl.p, sizeof host, cudaMemcpyDeviceToHost, s), "D2H");
    check(cudaStreamSynchronize(s), "sync");
    check_lookback(host.err, "BVH build");
    if (host.err) { why = "degenerate node (no finite SAH cost) or a leaf of 128+ triangles"; return 1; }
    return 0;
  };

  // phase 1
  const uint32_t max_small = T <= SUB ? 1u : T;  // a large node may shed one triangle per level
  TmpBuf<SmallTask> found(w, max_small), task(w, max_small);
  TmpBuf<uint32_t> big_start(w), big_off(w);
  TmpBuf<KBox> big_box(w);
  uint32_t n_lv = 0, n_small = 1, n_big = 0;
  if (T <= SUB) {
    k_one_task<<<1, 1, 0, s>>>(task.p, T, ctl.p);
  } else {
    const uint32_t max_nodes = T / SUB + 2, max_tiles = T / LV_TILE + max_nodes + 1;
    TmpBuf<uint4> fbox(w, 2 * (size_t)T);
    TmpBuf<LNode> node0(w, max_nodes), node1(w, max_nodes);
    TmpBuf<LTile> tile0(w, max_tiles), tile1(w, max_tiles);
    const size_t mt3 = 3 * (size_t)max_tiles;
    TmpBuf<FBox> tbox(w, mt3), carry0(w, mt3), carry1(w, mt3), nbox(w, max_nodes);
    TmpBuf<KBox> etbox(w, mt3), ecarry0(w, mt3), ecarry1(w, mt3), nexact(w, max_nodes);
    TmpBuf<uint32_t> nmin(w, 3 * (size_t)max_nodes), tmin(w, mt3), split(w, max_nodes), nleft(w, max_nodes),
        tcount(w, mt3);
    TmpBuf<float> cost(w, 3 * (size_t)T);
    TmpBuf<Best> best(w, mt3);
    TmpBuf<uint8_t> left(w, T);
    big_start.alloc(T);
    big_box.alloc(T);
    big_off.alloc((size_t)T + 1);
    k_frame<<<1, 1, 0, s>>>(ctl.p);
    k_round_boxes<<<blocks(T), 256, 0, s>>>(kbox.p, T, ctl.p, fbox.p);
    Level L{};
    L.ctl = ctl.p; L.kbox = kbox.p; L.fbox = fbox.p;
    L.A[0] = A[0]; L.A[1] = A[1];
    L.T = T; L.max_tiles = max_tiles;
    L.node[0] = node0.p; L.node[1] = node1.p; L.tile[0] = tile0.p; L.tile[1] = tile1.p;
    L.tbox = tbox.p; L.carry[0] = carry0.p; L.carry[1] = carry1.p;
    L.etbox = etbox.p; L.ecarry[0] = ecarry0.p; L.ecarry[1] = ecarry1.p;
    L.nbox = nbox.p; L.nmin = nmin.p; L.tmin = tmin.p; L.cost = cost.p; L.nexact = nexact.p; L.best = best.p;
    L.split = split.p; L.nleft = nleft.p; L.tcount = tcount.p; L.left = left.p;
    L.big_start = big_start.p; L.big_box = big_box.p; L.big_off = big_off.p; L.small = found.p;
    k_lv_start<<<8, 256, 0, s>>>(L, T);
    const unsigned tgrid = (unsigned)std::min<uint32_t>(3 * max_tiles, (uint32_t)sms * 8u);
    const unsigned ngrid = (unsigned)std::min<uint32_t>(blocks(3 * max_nodes * 32, LV_THREADS), (uint32_t)sms * 4u);
    uint32_t at_least = 1;  // levels that hold a large node whatever the splits
    while ((SUB << at_least) < T && at_least < 20) at_least++;
    for (;;) {
      const int b = (int)(n_lv & 1u);
      k_lv_reduce<<<tgrid, LV_THREADS, 0, s>>>(L, b);
      k_lv_carry<<<ngrid, LV_THREADS, 0, s>>>(L, b);
      k_lv_cost<<<tgrid, LV_THREADS, 0, s>>>(L, b);
      k_lv_exact_reduce<<<tgrid, LV_THREADS, 0, s>>>(L, b);
      k_lv_exact_carry<<<ngrid, LV_THREADS, 0, s>>>(L, b);
      k_lv_exact<<<tgrid, LV_THREADS, 0, s>>>(L, b);
      k_lv_decide<<<ngrid, LV_THREADS, 0, s>>>(L, b);
      k_lv_flag<<<tgrid, LV_THREADS, 0, s>>>(L, b);
      k_lv_count<<<tgrid, LV_THREADS, 0, s>>>(L, b);
      k_lv_offsets<<<ngrid, LV_THREADS, 0, s>>>(L, b);
      k_lv_scatter<<<tgrid, LV_THREADS, 0, s>>>(L, b);
      k_lv_next<<<1, NEXT_THREADS, 0, s>>>(L, b, n_lv);
      check(cudaGetLastError(), "bvh level");
      n_lv++;
      if (n_lv < at_least) continue;
      if (read_ctl()) return 1;
      if (!host.n_nodes) break;
    }
    n_small = host.n_small;
    n_big = host.n_big;
    TmpBuf<uint32_t> rank(w, T);
    check(cudaMemsetAsync(rank.p, 0, rank.bytes(), s), "memset");
    k_mark_tasks<<<blocks(n_small), 256, 0, s>>>(found.p, n_small, rank.p);
    scan_exclusive_u32(w, rank.p, rank.p, T, nullptr, err);
    k_place_tasks<<<blocks(n_small), 256, 0, s>>>(found.p, n_small, rank.p, task.p);
  }

  // phase 2
  TmpBuf<SubNode> sub_node(w, 2 * (size_t)T);
  TmpBuf<KBox> sub_box(w, 2 * (size_t)T);
  TmpBuf<uint32_t> leaf_ids(w, T), lv_inner(w, T), lv_leaf(w, T), depth(w, n_small), count(w, n_small);
  TmpBuf<uint16_t> local(w, T);
  Subtrees W{};
  W.ctl = ctl.p; W.kbox = kbox.p; W.A[0] = A[0]; W.A[1] = A[1]; W.T = T; W.task = task.p;
  W.node = sub_node.p; W.box = sub_box.p; W.leaf_ids = leaf_ids.p; W.lv_inner = lv_inner.p; W.lv_leaf = lv_leaf.p;
  W.depth = depth.p; W.count = count.p; W.local = local.p;
  check(cudaFuncSetAttribute(k_subtree, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(StShared)), "attr");
  k_subtree<<<n_small, ST_THREADS, sizeof(StShared), s>>>(W);
  check(cudaGetLastError(), "k_subtree");
  if (read_ctl()) return 1;
  const uint32_t n_nodes = 2 * (host.inner + n_big) + 1;
  if (n_nodes > 2 * T - 1) { why = "internal: node count"; return 1; }

  // #makeNormalizer(root.bounds) on the host, in double, JavaScript order
  double mn[3], mx[3];
  for (int a = 0; a < 3; a++) {
    auto val = [](i64 k) {
      const i64 u = k ^ ((k >> 63) & KEY_MAX);
      double d;
      std::memcpy(&d, &u, 8);
      return d;
    };
    mn[a] = val(host.root.mn[a]);
    mx[a] = val(host.root.mx[a]);
  }
  const Norm norm = make_norm(mn, mx);
  Columns C{};
  C.S = n_small;
  C.levels = host.levels;
  C.n_lv = n_lv;
  C.big_off = big_off.p;
  const size_t cells = (size_t)C.levels * C.S;
  TmpBuf<uint32_t> cn(w, cells), ci(w, cells), cl(w, cells), level_base(w, (size_t)C.levels + 1),
      leaf_off(w, (size_t)C.levels + 1);
  C.nodes = cn.p; C.inner = ci.p; C.leaf = cl.p; C.level_base = level_base.p; C.leaf_off = leaf_off.p;
  k_columns<<<C.levels, COL_THREADS, 0, s>>>(W, C);
  k_level_sums<<<1, COL_THREADS, 0, s>>>(C);
  out.nodes5.alloc(5 * (size_t)n_nodes);
  out.tri4_leaf.alloc(T);
  out.node_box.alloc(6 * (size_t)n_nodes);
  out.verts4.alloc(n_verts);
  const Emit E{tri4, norm, out.nodes5.p, out.tri4_leaf.p, reinterpret_cast<KBox*>(out.node_box.p), n_nodes, T, err};
  k_emit_small<<<n_small, 128, 0, s>>>(W, C, E, big_start.p);
  if (n_big) k_emit_large<<<blocks(n_big, 128), 128, 0, s>>>(W, C, E, big_start.p, big_box.p, n_big);
  launch_norm_verts(s, pos3, n_verts, norm, out.verts4.p);
  check(cudaGetLastError(), "bvh pack");
  if (read_ctl()) return 1;
  out.n_nodes = n_nodes;
  out.n_leaf_tris = T;
  out.depth = host.levels;
  for (int i = 0; i < 3; i++) out.norm[i] = norm.c[i];
  out.norm[3] = norm.scale;
  return 0;
}

}  // namespace pk
