// pk_cast.cu -- ray queries against the context's BVH on caller-owned device
// buffers: the GPU counterpart of the reference's CPU Raycaster used for
// autofocus (render/raycaster.js:114-131), with the closest-hit and any-hit
// semantics of trace.wgsl / trace_shadow.wgsl.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "../../include/pike.h"
#include "pk_ctx.h"
#include "pk_internal.cuh"
#include "pk_traverse.cuh"
#include "pk_util.h"

namespace pk {
namespace {

constexpr int CAST_THREADS = TRACE_THREADS;

// Every ray gets a record {t bits, triangle index or 0xffffffff, bary_mask, 0}.
//
// Large queries: persistent lanes (trace_lanes); any hit reports the closest
// triangle of the first leaf with a hit (trace_shadow.wgsl:154-158), so a leaf is
// always tested whole.
// Bound by the latency of dependent node and triangle fetches.  The grid fills
// the GPU whatever frame size the context is configured for (it used to be the
// frame's: 32 blocks for a 64x64 one).  2,097,143 incoherent closest-hit rays in
// the 1.3M-triangle scene: 13.3 ms -> 0.49 ms (4.3 Grays/s), 999,983 any-hit
// rays in 327,690 triangles: 3.52 -> 0.23 ms.  Rays sorted beforehand by octant
// and Morton code of the origin measured 0.46 and 0.20 ms, less than a sort
// would cost.
template <bool ANY>
__global__ void __launch_bounds__(CAST_THREADS, LANES_BLOCKS) k_cast(SceneDev sc, const float4* __restrict__ o4,
                                                                     const float4* __restrict__ d4, uint32_t n,
                                                                     uint4* __restrict__ hits4,
                                                                     uint32_t* __restrict__ ticket,
                                                                     uint32_t* __restrict__ err) {
  __shared__ int sstack[LANES_SMEM][CAST_THREADS];
  trace_lanes<ANY, true>(
      sc, n, ticket, err, sstack,
      [&](uint32_t j, float4& o, float4& d) {
        o = __ldcs(o4 + j);
        d = __ldcs(d4 + j);
      },
      [&](uint32_t j, float, float, float, float t, int i, uint32_t b) {
        __stcs(hits4 + j, make_uint4(__float_as_uint(t), (uint32_t)i, b, 0u));
      });
}

// Stable list of the rays that hit (increasing ray index) and its length, from
// the records' triangle indices: a lane per ray, tiles of LIST_TILE rays
// claimed in order, a warp-wide look-back per tile.
constexpr int LIST_THREADS = 256;
constexpr int LIST_WARPS = LIST_THREADS / 32;
constexpr int LIST_ROUNDS = 8;
constexpr uint32_t LIST_TILE = LIST_THREADS * LIST_ROUNDS;
__global__ void __launch_bounds__(LIST_THREADS) k_hit_list(const uint4* __restrict__ hits4, uint32_t n,
                                                            uint32_t* __restrict__ list, uint32_t* __restrict__ count,
                                                            uint32_t* __restrict__ ticket,
                                                            unsigned long long* __restrict__ tiles,
                                                            uint32_t* __restrict__ err, uint32_t* host_err) {
  __shared__ uint32_t s_tile, s_base;
  __shared__ uint32_t s_warp[LIST_WARPS];
  const uint32_t ntiles = (n + LIST_TILE - 1) / LIST_TILE;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, ltmask = (1u << lane) - 1u;
  if (ntiles == 0 && blockIdx.x == 0 && threadIdx.x == 0) *count = 0;
  for (;;) {
    if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    if (tile >= ntiles) break;
    const uint32_t j0 = tile * LIST_TILE + warp * (LIST_ROUNDS * 32u) + lane;
    uint32_t word[LIST_ROUNDS], mine = 0;
#pragma unroll
    for (int r = 0; r < LIST_ROUNDS; r++) {
      const uint32_t j = j0 + 32u * r;
      const bool hit = j < n && __ldg(&hits4[j].y) != 0xffffffffu;
      word[r] = __ballot_sync(0xffffffffu, hit);
      mine += (uint32_t)__popc(word[r]);
    }
    if (lane == 0) s_warp[warp] = mine;
    __syncthreads();
    uint32_t before = 0, total = 0;
#pragma unroll
    for (int k = 0; k < LIST_WARPS; k++) {
      if ((uint32_t)k < warp) before += s_warp[k];
      total += s_warp[k];
    }
    if (warp == 0) {
      const uint32_t e = unpack_a(lookback2_warp(tiles, tile, pack2(total, 0u), err));
      if (lane == 0) {
        s_base = e;
        if (tile == ntiles - 1) *count = e + total;
      }
    }
    __syncthreads();
    uint32_t at = s_base + before;
#pragma unroll
    for (int r = 0; r < LIST_ROUNDS; r++) {
      if ((word[r] >> lane) & 1u) list[at + __popc(word[r] & ltmask)] = j0 + 32u * r;
      at += (uint32_t)__popc(word[r]);
    }
    __syncthreads();
  }
  // every block sees the traversal's errors and its own look-back's
  if (threadIdx.x == 0 && *(volatile uint32_t*)err) *(volatile uint32_t*)host_err = 1u;
}

// Small queries (at most CAST_ONE rays): one launch of one block traces a ray
// per thread and lists the hits, since launches, memsets and a copy are most
// of such a query.  Where the line lies, one block against k_cast and k_hit_list,
// whole calls of pk_cast_rays_noalloc from Python in us, closest hits:
//   rays                                     257      512      768     1024
//   770 triangles, random rays            37  47   39  46   44  46   45  45
//   1,310,730 triangles, random           60  69   65  72   69  69   75  73
//   the same, one view                    35  43   36  44   46  45  180 176
//   524,288 loose triangles, random      222 190  249 207  273 212  305 210
//   the same, one view                   132 118  156 134  210 156  285 193
// Loose triangles are many steps a ray, and one SM does not hide their latency;
// even there a block of up to 512 rays is no slower than these queries were
// before it (244, 256, 254, 251 us; one view 154, 168, 206, 251).
constexpr uint32_t CAST_ONE = 512;
constexpr int ONE_SMEM = 8;
template <bool ANY>
__global__ void __launch_bounds__(CAST_ONE) k_cast_one(SceneDev sc, const float4* __restrict__ o4,
                                                       const float4* __restrict__ d4, uint32_t n,
                                                       uint4* __restrict__ hits4, uint32_t* __restrict__ list,
                                                       uint32_t* __restrict__ count, uint32_t* host_err) {
  __shared__ int sstack[ONE_SMEM][CAST_ONE];
  __shared__ uint32_t s_warp[CAST_ONE / 32];
  __shared__ uint32_t s_err;
  const uint32_t j = threadIdx.x, lane = j & 31u, warp = j >> 5;
  if (j == 0) s_err = 0;
  __syncthreads();
  bool hit = false;
  if (j < n) {
    const float4 o = o4[j], d = d4[j];
    float bt;
    int bi;
    uint32_t bb, nf = 0, nt = 0;
    traverse<ANY, false, (int)CAST_ONE, ONE_SMEM>(sc, o.x, o.y, o.z, d.x, d.y, d.z, bt, bi, bb, sstack, &s_err, nf, nt);
    hit = bi != -1;
    hits4[j] = make_uint4(__float_as_uint(bt), (uint32_t)bi, bb, 0u);
  }
  const uint32_t m = __ballot_sync(0xffffffffu, hit);
  if (lane == 0) s_warp[warp] = (uint32_t)__popc(m);
  __syncthreads();
  uint32_t before = 0, total = 0;
  for (uint32_t k = 0; k < blockDim.x / 32; k++) {
    if (k < warp) before += s_warp[k];
    total += s_warp[k];
  }
  if (hit) list[before + __popc(m & ((1u << lane) - 1u))] = j;
  if (j == 0) {
    *count = total;
    if (s_err) *(volatile uint32_t*)host_err = 1u;
  }
}

}  // namespace

// Scratch words the two kernels need for n rays: two tickets and an error
// word, and one look-back state per LIST_TILE rays; all start at zero.
struct CastScratch {
  uint32_t* tickets;  // [0] trace, [1] list, [2] error flags, [3] unused
  unsigned long long* tiles;
};
size_t cast_tiles(uint32_t n) { return ((size_t)n + LIST_TILE - 1) / LIST_TILE; }
size_t cast_bytes(uint32_t n) { return 16 + 8 * cast_tiles(n); }
// Queries of up to this many rays use 4 KB that the context keeps (taking the
// scratch from the pool: 4-5 us of a call).
constexpr uint32_t CAST_KEPT_RAYS = 1u << 20;
size_t cast_kept_bytes() { return cast_bytes(CAST_KEPT_RAYS); }  // pk_create

// The query on the context's stream; returns when it has finished.  `space`:
// cast_bytes(n) bytes of scratch when n > CAST_ONE.
int cast_run(pk_ctx* c, const char* what, const float4* o4, const float4* d4, uint32_t n, int any_hit, uint4* hits4,
             uint32_t* hit_index, uint32_t* n_hits, unsigned char* space) {
  const cudaStream_t st = c->stream;
  const SceneDev sc = c->dropin_scene();  // the drop-in's records whatever the trace mode
  volatile uint32_t* bad = c->host_words;
  *bad = 0;
  if (n <= CAST_ONE) {
    const unsigned threads = std::max(32u, (n + 31u) / 32u * 32u);
    if (any_hit) k_cast_one<true><<<1, threads, 0, st>>>(sc, o4, d4, n, hits4, hit_index, n_hits, c->host_words_dev);
    else k_cast_one<false><<<1, threads, 0, st>>>(sc, o4, d4, n, hits4, hit_index, n_hits, c->host_words_dev);
  } else {
    const CastScratch s{reinterpret_cast<uint32_t*>(space), reinterpret_cast<unsigned long long*>(space + 16)};
    check(cudaMemsetAsync(space, 0, cast_bytes(n), st), "memset");
    const unsigned warps = (unsigned)((n + 31) / 32);
    const unsigned grid = std::min((unsigned)c->sms * LANES_BLOCKS, (warps + CAST_THREADS / 32 - 1) / (CAST_THREADS / 32));
    if (any_hit) k_cast<true><<<grid, CAST_THREADS, 0, st>>>(sc, o4, d4, n, hits4, s.tickets, s.tickets + 2);
    else k_cast<false><<<grid, CAST_THREADS, 0, st>>>(sc, o4, d4, n, hits4, s.tickets, s.tickets + 2);
    const unsigned lgrid = (unsigned)std::min<size_t>(cast_tiles(n), (size_t)c->sms * 4);
    k_hit_list<<<lgrid, LIST_THREADS, 0, st>>>(hits4, n, hit_index, n_hits, s.tickets + 1, s.tiles, s.tickets + 2,
                                                c->host_words_dev);
  }
  check(cudaGetLastError(), what);
  check(cudaStreamSynchronize(st), "sync");
  if (*bad) {
    c->err = std::string(what) + ": device error flags";
    return PK_ERR_DEVICE;
  }
  return PK_OK;
}

}  // namespace pk

using namespace pk;

extern "C" int pk_cast_rays(pk_ctx* c, const float* ray_o4, const float* ray_d4, uint32_t n, int any_hit,
                            uint32_t* hits4, uint32_t* hit_index, uint32_t* n_hits) {
  if (!c) return PK_ERR_ARG;
  try {
    check(cudaSetDevice(c->device), "cudaSetDevice");
    if (!c->bvh_ready) { c->err = "pk_cast_rays: no BVH"; return PK_ERR_STATE; }
    if ((n && (!ray_o4 || !ray_d4 || !hits4 || !hit_index)) || !n_hits) { c->err = "pk_cast_rays: null buffer"; return PK_ERR_ARG; }
    if (n > (1u << 30)) { c->err = "pk_cast_rays: too many rays"; return PK_ERR_ARG; }
    const bool kept = n <= CAST_KEPT_RAYS;
    TmpBuf<unsigned char> space(c->scratch(), kept ? 0 : cast_bytes(n));
    return cast_run(c, "pk_cast_rays", reinterpret_cast<const float4*>(ray_o4), reinterpret_cast<const float4*>(ray_d4),
                    n, any_hit, reinterpret_cast<uint4*>(hits4), hit_index, n_hits, kept ? c->cast_space.p : space.p);
  } catch (CudaError& e) {
    c->err = e.what();
    return PK_ERR_CUDA;
  }
}

// ---- allocation-free variant -------------------------------------------------
// pk_cast_rays takes its scratch (work tickets and the look-back states of the
// hit list) for more than CAST_KEPT_RAYS rays from the context's pool, which can
// allocate.
// pk_cast_rays_noalloc takes it from the file-scope array below instead, so it
// allocates and frees nothing.  Every GPU that loads the library holds one copy
// of the array until the process exits.
namespace pk {
namespace {

constexpr uint32_t NOALLOC_MAX_RAYS = 1u << 20;  // rays per call
constexpr size_t NOALLOC_BYTES = 132352;         // as documented; the states of 2^20 rays take 4112
static_assert(16 + 8 * ((size_t)NOALLOC_MAX_RAYS / LIST_TILE) <= NOALLOC_BYTES, "scratch too small");

static __device__ __align__(256) unsigned char g_cast_scratch[NOALLOC_BYTES];

}  // namespace

// The array's device address on the current device.  In host code the name
// g_cast_scratch is only a host-side stand-in, not a device address, so
// pk_create looks the address up once, with the context's device current, and
// keeps it in the context: it stays valid exactly as long as the context's
// other device memory (a device reset invalidates both; the next pk_create
// looks it up again).
void* noalloc_scratch_address() {
  void* p = nullptr;
  check(cudaGetSymbolAddress(&p, g_cast_scratch), "cudaGetSymbolAddress(g_cast_scratch)");
  return p;
}

}  // namespace pk

extern "C" int pk_cast_rays_noalloc(pk_ctx* c, const float* ray_o4, const float* ray_d4, uint32_t n, int any_hit,
                                    uint32_t* hits4, uint32_t* hit_index, uint32_t* n_hits) {
  if (!c) return PK_ERR_ARG;
  try {
    check(cudaSetDevice(c->device), "cudaSetDevice");
    if (!c->bvh_ready) { c->err = "pk_cast_rays_noalloc: no BVH"; return PK_ERR_STATE; }
    if ((n && (!ray_o4 || !ray_d4 || !hits4 || !hit_index)) || !n_hits) {
      c->err = "pk_cast_rays_noalloc: null buffer";
      return PK_ERR_ARG;
    }
    if (n > NOALLOC_MAX_RAYS) {
      c->err = "pk_cast_rays_noalloc: at most 1048576 rays per call (the size of its static scratch)";
      return PK_ERR_ARG;
    }
    if (!c->cast_scratch) { c->err = "pk_cast_rays_noalloc: scratch address not set up"; return PK_ERR_STATE; }
    return cast_run(c, "pk_cast_rays_noalloc", reinterpret_cast<const float4*>(ray_o4),
                    reinterpret_cast<const float4*>(ray_d4), n, any_hit, reinterpret_cast<uint4*>(hits4), hit_index,
                    n_hits, static_cast<unsigned char*>(c->cast_scratch));
  } catch (CudaError& e) {
    c->err = e.what();
    return PK_ERR_CUDA;
  }
}

// ---- autofocus distance --------------------------------------------------------
// Raycaster.cast (render/raycaster.js:13-131): one ray traversed in double
// precision over the exact (unquantised) node bounds and normalised triangles,
// Möller-Trumbore with epsilon 1e-12, MAX_T = 1e6.  The recursion is kept as
// an explicit stack: closestNode orders the two children by entry distance,
// and each is entered only if its distance is below the closest hit found so
// far when its turn comes.  Math.min / Math.max propagate NaN, so a slab with
// 0 * inf culls the box exactly as the reference does.
namespace pk {
namespace {

__device__ __forceinline__ double jmin(double a, double b) {
  return (a != a || b != b) ? __longlong_as_double(0x7ff8000000000000ll) : (a < b ? a : (b < a ? b : (signbit(a) ? a : b)));
}
__device__ __forceinline__ double jmax(double a, double b) {
  return (a != a || b != b) ? __longlong_as_double(0x7ff8000000000000ll) : (a > b ? a : (b > a ? b : (signbit(a) ? b : a)));
}

struct FocusScene {
  const double* pos3;
  const int32_t* nodes5;
  const double* box6;
  const int4* tri4_leaf;
  double cx, cy, cz, s;
};

__device__ __forceinline__ double focus_box(const FocusScene& f, int node, const double* o, const double* inv) {
  const double* b = f.box6 + 6 * (size_t)node;
  const double c[3] = {f.cx, f.cy, f.cz};
  double t1[3], t2[3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const double mn = (b[a] - c[a]) * f.s, mx = (b[3 + a] - c[a]) * f.s;
    t1[a] = (mn - o[a]) * inv[a];
    t2[a] = (mx - o[a]) * inv[a];
  }
  double tmin = jmin(t1[0], t2[0]), tmax = jmax(t1[0], t2[0]);
  tmin = jmax(tmin, jmin(t1[1], t2[1]));
  tmax = jmin(tmax, jmax(t1[1], t2[1]));
  tmin = jmax(tmin, jmin(t1[2], t2[2]));
  tmax = jmin(tmax, jmax(t1[2], t2[2]));
  return (tmax >= tmin && tmax >= 0.0) ? tmin : 1000000.0;
}

__device__ __forceinline__ double focus_tri(const FocusScene& f, const int4 t4, const double* o, const double* d) {
  const double eps = 0.000000000001;
  double v[3][3];
  const int ids[3] = {t4.x, t4.y, t4.z};
  const double c[3] = {f.cx, f.cy, f.cz};
#pragma unroll
  for (int k = 0; k < 3; k++)
#pragma unroll
    for (int a = 0; a < 3; a++) v[k][a] = (f.pos3[3 * (size_t)ids[k] + a] - c[a]) * f.s;
  double e1[3], e2[3], tv[3];
#pragma unroll
  for (int a = 0; a < 3; a++) { e1[a] = v[1][a] - v[0][a]; e2[a] = v[2][a] - v[0][a]; tv[a] = o[a] - v[0][a]; }
  const double p[3] = {d[1] * e2[2] - d[2] * e2[1], -(d[0] * e2[2] - d[2] * e2[0]), d[0] * e2[1] - d[1] * e2[0]};
  const double det = 0.0 + e1[0] * p[0] + e1[1] * p[1] + e1[2] * p[2];
  if (det > -eps && det < eps) return 1000000.0;
  const double inv = 1.0 / det;
  const double u = (0.0 + tv[0] * p[0] + tv[1] * p[1] + tv[2] * p[2]) * inv;
  if (u < 0.0 || u > 1.0) return 1000000.0;
  const double q[3] = {tv[1] * e1[2] - tv[2] * e1[1], -(tv[0] * e1[2] - tv[2] * e1[0]), tv[0] * e1[1] - tv[1] * e1[0]};
  const double vv = (0.0 + d[0] * q[0] + d[1] * q[1] + d[2] * q[2]) * inv;
  if (vv < 0.0 || u + vv > 1.0) return 1000000.0;
  const double t = (0.0 + e2[0] * q[0] + e2[1] * q[1] + e2[2] * q[2]) * inv;
  return t > eps ? t : 1000000.0;
}

constexpr int FOCUS_STACK = 96;

__global__ void k_focus(FocusScene f, const double* __restrict__ rays6, uint32_t n, double* __restrict__ t_out,
                        uint32_t* __restrict__ err) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const double o[3] = {rays6[6 * r], rays6[6 * r + 1], rays6[6 * r + 2]};
  const double d[3] = {rays6[6 * r + 3], rays6[6 * r + 4], rays6[6 * r + 5]};
  const double inv[3] = {1.0 / d[0], 1.0 / d[1], 1.0 / d[2]};
  int stack_node[FOCUS_STACK];
  double stack_t[FOCUS_STACK];
  int sp = 0;
  double closest = 1000000.0;
  // the root is entered unconditionally (cast -> traverse(root, MAX_T))
  stack_node[sp] = 0;
  stack_t[sp] = -__longlong_as_double(0x7ff0000000000000ll);
  sp++;
  bool first = true;
  while (sp > 0) {
    --sp;
    const int node = stack_node[sp];
    if (!first && !(stack_t[sp] < closest)) continue;
    first = false;
    const int32_t* nd = f.nodes5 + 5 * (size_t)node;
    if (nd[1] > -1) {  // leaf: processLeaf returns the leaf's own minimum
      const int size = nd[1] >> 24, base = nd[1] & 0x00ffffff;
      double res = 1000000.0;
      for (int i = 0; i < size; i++) {
        const double x = focus_tri(f, f.tri4_leaf[base + i], o, d);
        if (x < res) res = x;
      }
      closest = jmin(res, closest);
      continue;
    }
    const int l = nd[0], rr = nd[0] + 1;
    const double tl = focus_box(f, l, o, inv), tr = focus_box(f, rr, o, inv);
    // closestNode: a child whose box is missed is dropped; the nearer one goes first
    const int ln = tl < 1000000.0 ? l : -1, rn = tr < 1000000.0 ? rr : -1;
    int o0, o1;
    double t0, t1;
    if (tl < tr) { o0 = ln; t0 = tl; o1 = rn; t1 = tr; } else { o0 = rn; t0 = tr; o1 = ln; t1 = tl; }
    if (sp + 2 > FOCUS_STACK) { atomicOr(err, 1u); break; }
    if (o1 >= 0) { stack_node[sp] = o1; stack_t[sp] = t1; sp++; }
    if (o0 >= 0) { stack_node[sp] = o0; stack_t[sp] = t0; sp++; }
  }
  t_out[r] = closest;
}

}  // namespace
}  // namespace pk

extern "C" int pk_focus_distance(pk_ctx* c, const double origin[3], const double dir[3], double* t_out,
                                 double* focal_depth_out) {
  if (!c) return PK_ERR_ARG;
  try {
    check(cudaSetDevice(c->device), "cudaSetDevice");
    if (!c->bvh_ready || !c->node_box_d.p || c->norm[3] == 0.0) {
      c->err = "pk_focus_distance: needs a BVH built by pk_bvh_build (its exact node bounds)";
      return PK_ERR_STATE;
    }
    if (!origin || !dir || !t_out) { c->err = "pk_focus_distance: null argument"; return PK_ERR_ARG; }
    const double ray[6] = {origin[0], origin[1], origin[2], dir[0], dir[1], dir[2]};
    DevBuf<double> dray(6), dt(1);
    DevBuf<uint32_t> err(1);
    check(cudaMemsetAsync(err.p, 0, 4, c->stream), "memset");
    check(cudaMemcpyAsync(dray.p, ray, sizeof ray, cudaMemcpyHostToDevice, c->stream), "H2D");
    const FocusScene f{c->pos.p, c->nodes5.p, c->node_box_d.p, reinterpret_cast<const int4*>(c->tri4_leaf.p),
                       c->norm[0], c->norm[1], c->norm[2], c->norm[3]};
    k_focus<<<1, 32, 0, c->stream>>>(f, dray.p, 1, dt.p, err.p);
    check(cudaGetLastError(), "k_focus");
    double t = 0.0;
    uint32_t e = 0;
    check(cudaMemcpyAsync(&t, dt.p, 8, cudaMemcpyDeviceToHost, c->stream), "D2H");
    check(cudaMemcpyAsync(&e, err.p, 4, cudaMemcpyDeviceToHost, c->stream), "D2H");
    check(cudaStreamSynchronize(c->stream), "sync");
    if (e) { c->err = "pk_focus_distance: traversal stack overflow"; return PK_ERR_DEVICE; }
    *t_out = t;
    if (focal_depth_out) *focal_depth_out = 1.0 - 1.0 / t;  // PikeRenderer.focusCamera (pike.js:88-90)
    return PK_OK;
  } catch (CudaError& e) {
    c->err = e.what();
    return PK_ERR_CUDA;
  }
}
