// pk_traverse.cuh -- binary-BVH traversal of trace.wgsl / trace_shadow.wgsl
// on the traversal-format BVH (see SceneDev in pk_internal.cuh).
#pragma once
#include "pk_internal.cuh"

namespace pk {

constexpr float MAX_T = 100000.0f;

// =====================================================================
// trace.wgsl:83-189 / trace_shadow.wgsl:82-190: BVH traversal.
// =====================================================================
// Both planes of the axes come as pairs {x, y} and {z, z} for the packed FP32
// instructions, which round each half like the single ones and issue once for
// two: 12 instead of 24 subtractions and multiplications per inner node.  The
// traversals issue on half of the cycles and stall mostly on latency, so this
// gives less than its share of the instructions (eight 1080p frames 25.8 ->
// 25.4 ms, 16 batched requests 29.1 -> 28.4 ms; z apart, without the doubled
// registers of {oz, oz} and {iz, iz}: 25.5 and 28.5).
// (b - o) * i of both halves
__device__ __forceinline__ float2 pair_dist(F2 b, F2 o, F2 i) {
  float2 r;
  asm("{\n\t.reg .b64 t;\n\tsub.rn.f32x2 t, %2, %3;\n\tmul.rn.f32x2 t, t, %4;\n\tmov.b64 {%0, %1}, t;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "l"(b), "l"(o), "l"(i));
  return r;
}
// t1: distances {x, y} of the x_range.x, y_range.x bounds (quantised max), t2 of
// the .y bounds (min), z both.  True where trace.wgsl's box distance is below
// `best`: a box that is hit has the distance tmin, one that is not MAX_T, which
// no best distance exceeds.  (Returning the distance and comparing it outside:
// 24.0 against 23.7 ms.)
__device__ __forceinline__ bool box_entry(float2 t1, float2 t2, float2 z, float best, float& tmin) {
  // fminf/fmaxf agree with minNum/maxNum except for the sign of a zero
  // result, which only ever feeds comparisons here.  (Three-input min/max
  // measured the same: 23.64-23.73 against 23.69-23.76 ms for eight 1080p frames.)
  const float tmax = fminf(fminf(fmaxf(t1.x, t2.x), fmaxf(t1.y, t2.y)), fmaxf(z.x, z.y));
  tmin = fmaxf(fmaxf(fminf(t1.x, t2.x), fminf(t1.y, t2.y)), fminf(z.x, z.y));
  return tmax >= tmin && tmax > 0.0f && tmin < best;
}

// unpack2x16snorm component: max(s / 32767, -1), the value the reference decode
// and the 64-byte records hold (the tests check all 65536).
__device__ __forceinline__ float snorm16_decode(int s) { return snorm16(s); }
__device__ __forceinline__ float snorm_lo(int m) { return snorm16_decode((int)(int16_t)(uint16_t)((uint32_t)m & 0xffffu)); }
__device__ __forceinline__ float snorm_hi(int m) { return snorm16_decode((int)(int16_t)(uint16_t)((uint32_t)m >> 16)); }

// trace.wgsl:97-114: Moller-Trumbore on one leaf-ordered triangle record
// {v0.xyz, e1.x}{e1.yz, e2.xy}{e2.z}.  Returns false where the reference
// `continue`s (parallel ray, u or v outside the triangle); otherwise res = the
// distance when it exceeds eps, else MAX_T.
__device__ __forceinline__ bool mt_test(const SceneDev& sc, int idx, float ox, float oy, float oz, float dx,
                                        float dy, float dz, float eps, float& res, float& u, float& v) {
  const float4* tp = sc.tris + 3 * (size_t)idx;
  const float4 A = __ldg(tp), B = __ldg(tp + 1), Cc = __ldg(tp + 2);
  const float e1x = A.w, e1y = B.x, e1z = B.y, e2x = B.z, e2y = B.w, e2z = Cc.x;
  const float px = dy * e2z - dz * e2y, py = dz * e2x - dx * e2z, pz = dx * e2y - dy * e2x;
  const float det = e1x * px + e1y * py + e1z * pz;
  if (fabsf(det) < eps) return false;
  const float inv_det = 1.0f / det;
  const float tx = ox - A.x, ty = oy - A.y, tz = oz - A.z;
  u = (tx * px + ty * py + tz * pz) * inv_det;
  if (u < 0.0f || u > 1.0f) return false;
  const float qx = ty * e1z - tz * e1y, qy = tz * e1x - tx * e1z, qz = tx * e1y - ty * e1x;
  v = (dx * qx + dy * qy + dz * qz) * inv_det;
  if (v < 0.0f || u + v > 1.0f) return false;
  const float dist = (e2x * qx + e2y * qy + e2z * qz) * inv_det;
  res = dist > eps ? dist : MAX_T;
  return true;
}

constexpr int TRACE_THREADS = 128;
constexpr int STACK_SMEM = 32;   // per-thread entries kept in shared memory
// (traverse_rt keeps the remaining 64 - SSTACK entries in local memory)

// One inner-node step: both children's entry distances and child codes.
// COMPACT: 32-byte records keep the reference's snorm16 boxes {Lx, Ly, Lz, Rx}{Ry, Rz,
// codeL, codeR}; 64-byte records (the default: fewer instructions per step,
// which matters more than bytes here) hold the same boxes decoded.
// (Prefetching both children's records into L1 while the boxes are tested
// measured far slower at 1080p: 3188-3197 Mrays/s against 3738-3746, and
// 2766-2769 with the leaves' first triangle too.)
template <bool COMPACT>
__device__ __forceinline__ void inner_children(const SceneDev& sc, int cur, float ox, float oy, float oz, float ix,
                                               float iy, float iz, float best, bool& lok, bool& rok, float& lh,
                                               float& rh, int& cl, int& cr) {
  const F2 o = pair_of(ox, oy), i = pair_of(ix, iy), oo = pair_of(oz, oz), ii = pair_of(iz, iz);
  if (COMPACT) {
    const int4* rec = sc.inner32 + 2 * (size_t)cur;
    const int4 q0 = __ldg(rec), q1 = __ldg(rec + 1);
    lok = box_entry(pair_dist(pair_of(snorm_lo(q0.x), snorm_lo(q0.y)), o, i),
                   pair_dist(pair_of(snorm_hi(q0.x), snorm_hi(q0.y)), o, i),
                   pair_dist(pair_of(snorm_lo(q0.z), snorm_hi(q0.z)), oo, ii), best, lh);
    rok = box_entry(pair_dist(pair_of(snorm_lo(q0.w), snorm_lo(q1.x)), o, i),
                   pair_dist(pair_of(snorm_hi(q0.w), snorm_hi(q1.x)), o, i),
                   pair_dist(pair_of(snorm_lo(q1.y), snorm_hi(q1.y)), oo, ii), best, rh);
    cl = q1.z;
    cr = q1.w;
  } else {  // {Lx0, Ly0, Lx1, Ly1}{Lz0, Lz1, Rz0, Rz1}{Rx0, Ry0, Rx1, Ry1}{codeL, codeR, -, -}
    const ulonglong2* rec = reinterpret_cast<const ulonglong2*>(sc.inner + 4 * (size_t)cur);
    const ulonglong2 a = __ldg(rec), b = __ldg(rec + 1), c = __ldg(rec + 2);
    const int4 ch = __ldg(reinterpret_cast<const int4*>(rec) + 3);
    lok = box_entry(pair_dist(a.x, o, i), pair_dist(a.y, o, i), pair_dist(b.x, oo, ii), best, lh);
    rok = box_entry(pair_dist(c.x, o, i), pair_dist(c.y, o, i), pair_dist(b.y, oo, ii), best, rh);
    cl = ch.x;
    cr = ch.y;
  }
}

// BLOCK threads per block share `sstack` (SSTACK entries per thread in shared
// memory, 64 - SSTACK more in local memory).  ANY: any hit (trace_shadow.wgsl)
// rather than closest hit; a constant at every inlined call site, a run-time
// value where one out-of-line copy serves both.
template <bool COUNT, int BLOCK, int SSTACK, bool COMPACT = false>
__device__ __forceinline__ void traverse_rt(const bool ANY, const SceneDev& sc, float ox, float oy, float oz,
                                            float dx, float dy, float dz, float& best_t, int& best_i,
                                            uint32_t& best_b, int (*sstack)[BLOCK], uint32_t* err,
                                            uint32_t& nfetch, uint32_t& ntest) {
  const float eps = ANY ? 1e-7f : 1e-8f;
  const float ix = 1.0f / dx, iy = 1.0f / dy, iz = 1.0f / dz;
  constexpr int LOCAL = 64 - SSTACK;  // 64 entries in all
  int lstack[LOCAL];
  const int tid = threadIdx.x;
  int sp = 0;
  int cur = sc.root;
  best_t = MAX_T;
  best_i = -1;
  best_b = 0u;
  for (;;) {
    if (cur >= 0) {
      if (COUNT) nfetch += 3;
      float lh, rh;
      bool lok, rok;
      int cl, cr;
      inner_children<COMPACT>(sc, cur, ox, oy, oz, ix, iy, iz, best_t, lok, rok, lh, rh, cl, cr);
      if (lok && rok) {
        int nearc, farc;
        if (lh > rh) { nearc = cr; farc = cl; } else { nearc = cl; farc = cr; }
        if (sp < SSTACK) sstack[sp][tid] = farc;
        else if (sp < SSTACK + LOCAL) lstack[sp - SSTACK] = farc;
        else { atomicOr(err, ERR_STACK); break; }
        ++sp;
        cur = nearc;
        continue;
      }
      if (lok) { cur = cl; continue; }
      if (rok) { cur = cr; continue; }
    } else {
      if (COUNT) nfetch += 1;
      const uint32_t word = (uint32_t)cur & 0x7fffffffu;
      const int size = (int)(word >> 24);
      const int base = (int)(word & 0x00ffffffu);
      for (int i = 0; i < size; i++) {
        if (COUNT) ntest += 1;
        float res, u, v;
        if (!mt_test(sc, base + i, ox, oy, oz, dx, dy, dz, eps, res, u, v)) continue;
        if (res < best_t) {
          best_t = res;
          best_i = base + i;
          best_b = pack_unorm16(u) | (pack_unorm16(v) << 16);
        }
      }
      if (ANY && best_i != -1) break;
    }
    if (sp == 0) break;
    --sp;
    cur = sp < SSTACK ? sstack[sp][tid] : lstack[sp - SSTACK];
  }
}
template <bool ANY, bool COUNT, int BLOCK = TRACE_THREADS, int SSTACK = STACK_SMEM, bool COMPACT = false>
__device__ __forceinline__ void traverse(const SceneDev& sc, float ox, float oy, float oz, float dx, float dy,
                                         float dz, float& best_t, int& best_i, uint32_t& best_b,
                                         int (*sstack)[BLOCK], uint32_t* err, uint32_t& nfetch,
                                         uint32_t& ntest) {
  traverse_rt<COUNT, BLOCK, SSTACK, COMPACT>(ANY, sc, ox, oy, oz, dx, dy, dz, best_t, best_i, best_b, sstack, err, nfetch,
                                    ntest);
}

// Persistent lanes over n rays, for kernels of TRACE_THREADS threads.  A lane
// owns one ray at a time; when at least LANES_REFILL lanes of a warp are idle
// they claim new rays together from `ticket` (zero at launch), and a lane takes
// at most LANES_BUDGET inner steps before the warp meets again, so no lane
// waits for the longest of a fixed group of 32 rays.  No speculation: each ray
// visits the nodes and leaves of trace.wgsl's (trace_shadow.wgsl's) loop in its
// order.  WHOLE: an any-hit ray tests the leaf it hits in to its end, for
// callers that want the triangle; otherwise it stops at the first accepted one.
// load(j, o, d) fetches ray j; done(j, d, t, triangle, barycentrics) takes the
// result (triangle -1: none).
// (Threshold, budget, stack split and leaf loop as measured for the frame's
// traversal, k_trace_dyn; 2,097,143 random rays: leaf loop unrolled by 4 476 us,
// not unrolled 463, without the 32-byte records' code 450.  Handing results in
// at the next refill instead of at once: 533.)
constexpr int LANES_REFILL = 16;
constexpr int LANES_BUDGET = 8;
constexpr int LANES_SMEM = 8;  // stack entries per lane in shared memory, the rest of 64 in local memory
constexpr int LANES_LOCAL = 64 - LANES_SMEM;
constexpr int LANES_BLOCKS = 10;  // resident blocks per SM (48 registers)

template <bool ANY, bool WHOLE, class Load, class Done>
__device__ __forceinline__ void trace_lanes(const SceneDev& sc, uint32_t n, uint32_t* __restrict__ ticket,
                                            uint32_t* err, int (*sstack)[TRACE_THREADS], Load load, Done done) {
  int lstack[LANES_LOCAL];
  const int lane = threadIdx.x & 31, tid = threadIdx.x;
  const uint32_t ltmask = (1u << lane) - 1u;
  const float eps = ANY ? 1e-7f : 1e-8f;
  uint32_t j = 0;
  bool have = false, exhausted = false;
  float ox = 0.f, oy = 0.f, oz = 0.f, dx = 0.f, dy = 0.f, dz = 0.f, ix = 0.f, iy = 0.f, iz = 0.f;
  float best_t = MAX_T;
  int best_i = -1;
  uint32_t best_b = 0u;
  int sp = 0, cur = 0;
  for (;;) {
    const uint32_t idle = __ballot_sync(0xffffffffu, !have && !exhausted);
    const uint32_t busy = __ballot_sync(0xffffffffu, have);
    if (idle && (__popc(idle) >= LANES_REFILL || busy == 0u)) {
      const int leader = __ffs(idle) - 1;
      uint32_t base = 0;
      if (lane == leader) base = atomicAdd(ticket, (uint32_t)__popc(idle));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (!have && !exhausted) {
        j = base + (uint32_t)__popc(idle & ltmask);
        if (j < n) {
          float4 o, d;
          load(j, o, d);
          ox = o.x; oy = o.y; oz = o.z;
          dx = d.x; dy = d.y; dz = d.z;
          ix = 1.0f / dx; iy = 1.0f / dy; iz = 1.0f / dz;
          best_t = MAX_T; best_i = -1; best_b = 0u;
          sp = 0;
          cur = sc.root;
          have = true;
        } else {
          exhausted = true;
        }
      }
    }
    if (!__any_sync(0xffffffffu, have)) break;
    if (!have) continue;
    bool fin = false;
    int budget = LANES_BUDGET;
    while (cur >= 0 && budget-- > 0) {
      float lh, rh;
      bool lok, rok;
      int cl, cr;
      inner_children<false>(sc, cur, ox, oy, oz, ix, iy, iz, best_t, lok, rok, lh, rh, cl, cr);
      if (lok && rok) {
        int nearc, farc;
        if (lh > rh) { nearc = cr; farc = cl; } else { nearc = cl; farc = cr; }
        if (sp < LANES_SMEM) sstack[sp][tid] = farc;
        else if (sp < LANES_SMEM + LANES_LOCAL) lstack[sp - LANES_SMEM] = farc;
        else { atomicOr(err, ERR_STACK); fin = true; break; }
        ++sp;
        cur = nearc;
        continue;
      }
      if (lok) { cur = cl; continue; }
      if (rok) { cur = cr; continue; }
      if (sp == 0) { fin = true; break; }
      --sp;
      cur = sp < LANES_SMEM ? sstack[sp][tid] : lstack[sp - LANES_SMEM];
    }
    while (!fin && cur < 0) {
      const uint32_t word = (uint32_t)cur & 0x7fffffffu;
      const int size = (int)(word >> 24);
      const int base = (int)(word & 0x00ffffffu);
#pragma unroll 1
      for (int i = 0; i < size; i++) {
        float res, u, v;
        if (!mt_test(sc, base + i, ox, oy, oz, dx, dy, dz, eps, res, u, v)) continue;
        if (res < best_t) {
          best_t = res;
          best_i = base + i;
          best_b = pack_unorm16(u) | (pack_unorm16(v) << 16);
        }
        if (ANY && !WHOLE && best_i != -1) break;
      }
      if (ANY && best_i != -1) { fin = true; break; }
      if (sp == 0) { fin = true; break; }
      --sp;
      cur = sp < LANES_SMEM ? sstack[sp][tid] : lstack[sp - LANES_SMEM];
    }
    if (fin) {
      done(j, dx, dy, dz, best_t, best_i, best_b);
      have = false;
    }
  }
}

}  // namespace pk
