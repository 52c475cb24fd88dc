// pk_diff.cu -- form (3): the path-replay adjoint of the drop-in's estimator.
//
// No reference counterpart (the reference has no differentiation).  The
// forward pass renders, path by path, the estimator the drop-in's passes
// render: camera.wgsl's ray (the context's camera and sample index),
// trace.wgsl closest hits and trace_shadow.wgsl any hits on the drop-in's
// records, shade_hit.wgsl:407-483 at every hit (GGX VNDF sampling of a
// microfacet normal, the Fresnel lobe choice between Lambert and specular, the
// bounce ray weighted by the power heuristic against the environment pdf,
// next-event estimation of the environment with both lobes MIS-weighted) and
// shade_miss.wgsl's environment radiance for rays that leave.  Base colour,
// roughness and metallic come from per-material FP32 parameters instead of
// the atlas (normal map, opacity and emission still come from it), and the
// environment radiance from an FP32 RGB equirect map.  As in pk_batch, the
// shading random numbers are seeded with the bounce index where the wavefront
// uses the hit-queue slot (shade_hit.wgsl:421), so the images equal the
// drop-in's in distribution.
//
// Detached sampling.  Paths are sampled with the sampling roughness rho0 and
// with the environment tables of pk_diff_set_env_sampling, both held fixed,
// and every path is weighted by
//     prod_v V(m_v; alpha_v) / V(m_v; alpha0_v)  x  (the drop-in's weights at theta),
// V(m; a) = G1(wo, m; a) D(m; a) being the density of the sampled microfacet
// normal m up to factors that cancel (Heitz's VNDF; the ratio is taken as 1
// where that density does not apply, wo below the shading hemisphere).  At theta = theta0 every
// ratio is exactly 1 and the arithmetic is the drop-in's operation for
// operation; for any theta the weighted path is an importance-sampled
// estimate of the drop-in's expected image at theta, so its derivative at
// theta0 is an unbiased estimate of the image gradient: the derivative of the
// weights along the fixed path plus the score d log V / d alpha of every
// sampled normal.  The lobe choice depends on metallic only, which is not
// differentiated; the environment sampling tables, and the pdfs they give the
// MIS weights, are held fixed.  For fixed seeds and theta0 the estimator is a
// smooth function of theta (paths do not move), so its exact derivative is
// what central differences with common random numbers measure.
//
// Adjoint.  The backward pass replays every path from its seed (nothing is
// stored between the passes; k_path_*<true>) and records per vertex the throughput T that
// reaches it, the factor P to the next vertex's throughput, the contribution
// factor Q of the vertex (next-event estimate, emission, or the environment
// when the ray leaves) and their derivatives; a backward sweep with
// L_v = Q_v + P_v L_{v+1} gives
//     dLoss/dtheta_v = sum_c g_c T_v,c (dQ_v,c + dP_v,c L_{v+1},c),
//     dLoss/dE_c(texel of v) = g_c T_v,c dQ_v,c/dE_c.
// Material terms go through warp-aggregated atomics into per-block FP32
// partials in shared memory, flushed with FP64 atomics; environment terms are
// warp-aggregated per texel and added in FP64.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <string>

#include "../../include/pike.h"
#include "pk_ctx.h"
#include "pk_math.cuh"
#include "pk_shade.cuh"
#include "pk_traverse.cuh"

namespace pk {

constexpr int DIFF_MAX_DEPTH = 8;

struct DiffParams {
  const float* albedo;  // n_mats x 3 (base colour)
  const float* rough;   // roughness the weights are evaluated with
  const float* rough0;  // roughness the normals are sampled with
  const float* metal;
  uint32_t n_mats;
  const float* env;     // env_h x env_w x 3
  int env_w, env_h;
  int spp, depth;
  uint32_t sample_base;
};

// A unit direction's y component can round to just above 1 in magnitude,
// where acos (and with it envPdf in the drop-in) is NaN and the NaN poisons
// the pixel; the differentiable renderer clamps y to [-1, 1] in its
// environment lookups (the texel chosen is the one the drop-in reads).
__device__ __forceinline__ V3 clamp_y(V3 d) { return v3(d.x, fmin_(fmax_(d.y, -1.0f), 1.0f), d.z); }

// shade_miss.wgsl's texel choice (env_color) on the FP32 map; tex = its index.
__device__ __forceinline__ V3 diff_env(const DiffParams& P, float theta, V3 dir, int& tex) {
  dir = clamp_y(dir);
  const float u = theta + atan2_(dir.z, dir.x) / c::TAU;
  const float v = acos_(dir.y) * c::INV_PI;
  const int x = wrap_floor(u * (float)P.env_w, P.env_w), y = wrap_floor(v * (float)P.env_h, P.env_h);
  tex = y * P.env_w + x;
  const float* e = P.env + 3 * (size_t)tex;
  return v3(__ldg(e), __ldg(e + 1), __ldg(e + 2));
}

// d log D(m; a) / da of shade_hit.wgsl's GGX_D with au = av = a:
// D = 1 / (pi a^2 ell^2), ell = q / a^2 + mz^2, q = mx^2 + my^2.
__device__ __forceinline__ float dlog_ggx_d(V3 m, float a) {
  const float q = m.x * m.x + m.y * m.y, z = a * a * m.z * m.z;
  return 2.0f * (q - z) / (a * (q + z));
}
// d log G1(w, m; a) / da of GGX_G1: G1 = 2 / (1 + s), s = sqrt(1 + a^2 k),
// k = (wx^2 + wy^2) / wz^2; 0 where GGX_G1 is 0.
__device__ __forceinline__ float dlog_ggx_g1(V3 w, V3 m, float a) {
  if (dot(w, m) * w.z <= 0.0f) return 0.0f;
  const float k = (w.x * w.x + w.y * w.y) / (w.z * w.z);
  const float s = sqrtf(1.0f + a * a * k);
  return -a * k / (s * (1.0f + s));
}
// d/dp0 of the power heuristic p0^2 / (p0^2 + p1^2).
__device__ __forceinline__ float dph_dp0(float p0, float p1) {
  const float d = p0 * p0 + p1 * p1;
  if (!(d > 0.0f) || !isfinite(d)) return 0.0f;
  return 2.0f * (p0 / d) * (p1 * p1 / d);
}

// One shading event (shade_hit.wgsl main for one hit) with the material's
// parameters.  For the adjoint (DERIV) also the bounce factor P (bt = t4 * P),
// the shadow factor S (st = t4 * S) and the emission factor Qem (em = t4 *
// Qem), with their derivatives by the hit material's albedo (per channel, of
// the same channel) and roughness.
struct DiffShade {
  bool emitted, eb, es, pass;  // pass: the alpha pass-through (the ray goes on unchanged)
  V3 em;
  float4 bo, bd, bt, so, sd, st;
  V3 P, dPa, dPr, S, dSa, dSr, Qem;
  int mat;
};

template <bool DERIV>
__device__ __forceinline__ void shade_diff(const SceneDev& sc, const EnvDev& env, const DiffParams& P, float theta,
                                           int32_t samples, uint32_t r, float4 o4, float4 d4, float4 t4, uint4 hr,
                                           DiffShade& out) {
  const V3 zero = v3(0.0f, 0.0f, 0.0f);
  out.emitted = out.eb = out.es = out.pass = false;
  out.em = out.P = out.dPa = out.dPr = out.S = out.dSa = out.dSr = out.Qem = zero;
  const V3 ro = v3(o4.x, o4.y, o4.z), rd = v3(d4.x, d4.y, d4.z);
  const float ht = __uint_as_float(hr.x);
  const uint32_t mask = __float_as_uint(t4.w);
  const uint32_t color_idx = mask & 0x0fffffffu;
  const uint32_t ray_type = mask & 0xf0000000u;
  Hash h;
  h.seed = (r * 1973u + color_idx * 9277u + (uint32_t)samples * 26699u) | 1u;
  h.seed = h.next();
  SI si = surface(sc, ro, rd, ht, (int)hr.y, hr.z);
  int mat = __ldg(sc.tri4 + hr.y).w;
  if ((uint32_t)mat >= sc.n_mats) mat = 0;  // surface()'s clamp
  out.mat = mat;
  const float rho = __ldg(P.rough + mat), rho0 = __ldg(P.rough0 + mat), mu = __ldg(P.metal + mat);
  si.base = v3(__ldg(P.albedo + 3 * mat), __ldg(P.albedo + 3 * mat + 1), __ldg(P.albedo + 3 * mat + 2));
  si.metallic = mu;
  si.alpha = rho * rho;
  si.spec = v3(mix1(1.0f, si.base.x, mu), mix1(1.0f, si.base.y, mu), mix1(1.0f, si.base.z, mu));
  if (h.rand() > si.opacity) {  // alpha pass-through: same direction and throughput
    const V3 ao = add(ro, scale(rd, ht + SHADE_EPS * 40.0f));
    out.eb = out.pass = true;
    out.bo = make_float4(ao.x, ao.y, ao.z, 0.0f);
    out.bd = d4;
    out.bt = t4;
    out.P = v3(1.0f, 1.0f, 1.0f);
    return;
  }
  if (dot(si.emission, v3(1.0f, 1.0f, 1.0f)) > 0.0f) {
    const float att = fmax_(dot(si.n, matvec(si.b1, si.b2, si.n, si.wo)), 0.0f);
    out.em = v3(50.0f * si.emission.x * t4.x * att, 50.0f * si.emission.y * t4.y * att,
                50.0f * si.emission.z * t4.z * att);
    out.Qem = v3(50.0f * si.emission.x * att, 50.0f * si.emission.y * att, 50.0f * si.emission.z * att);
    out.emitted = true;
    return;
  }
  if (ray_type == 0x10000000u) return;
  SI s0 = si;
  s0.alpha = rho0 * rho0;
  const V3 m = sample_ggx(h, s0);
  const float f = mix1(schlick(fmax_(dot(si.wo, m), 0.0f), 1.5f), 1.0f, si.metallic);
  const float a = si.alpha;
  // V(m; a) / V(m; a0): exactly 1 when the two roughness values agree, and
  // taken as 1 where the VNDF density does not apply (G1(wo, m) = 0: the
  // view direction below the shading hemisphere)
  const bool vndf = dot(si.wo, m) * si.wo.z > 0.0f;
  float ratio = 1.0f;
  if (vndf && s0.alpha != a)
    ratio = (ggx_g1(si.wo, m, a, a) * ggx_d(m, a, a)) / (ggx_g1(si.wo, m, s0.alpha, s0.alpha) * ggx_d(m, s0.alpha, s0.alpha));
  const float dlv = DERIV && vndf ? dlog_ggx_d(m, a) + dlog_ggx_g1(si.wo, m, a) : 0.0f;
  const float dadr = 2.0f * rho;  // d alpha / d roughness
  Sample bs;
  V3 bsdf, hb;  // hb: the specular bounce's half vector
  bool lamb;
  if (h.rand() > f) {
    const float lr = sqrtf(h.rand());
    const float lphi = c::TAU * h.rand();
    const SinCos lp = sincos_(lphi);
    const float x = lr * lp.c;
    const float y = lr * lp.s;
    const float z = sqrtf(fmax_(0.0f, 1.0f - x * x - y * y));
    bs.wi = v3(x, y, z);
    bs.pdf = lambert_pdf(bs.wi);
    bsdf = eval_lambert(si, bs);
    lamb = true;
  } else {
    bs.wi = reflect(neg(si.wo), m);
    bs.pdf = specular_pdf(si, m);
    hb = normalize(add(si.wo, bs.wi));
    bsdf = eval_specular(si, bs, hb);
    lamb = false;
  }
  if (bs.wi.z > 0.0f) {
    const V3 dir = matvec(si.b1, si.b2, si.n, bs.wi);
    const float pe = env.enabled ? env_pdf_dir(env, theta, clamp_y(dir)) : 0.0f;
    const float weight = env.enabled ? power_heuristic(bs.pdf, pe) : 1.0f;
    out.eb = true;
    out.bo = make_float4(si.origin.x, si.origin.y, si.origin.z, 0.0f);
    out.bd = make_float4(dir.x, dir.y, dir.z, 0.0f);
    out.bt = make_float4(bsdf.x * t4.x * weight * ratio, bsdf.y * t4.y * weight * ratio,
                         bsdf.z * t4.z * weight * ratio, t4.w);
    if (DERIV) {
      out.P = v3(bsdf.x * weight * ratio, bsdf.y * weight * ratio, bsdf.z * weight * ratio);
      if (lamb) {  // base * INV_PI * max(eps, wi.z) / pdf; nothing else depends on theta
        const float k1 = c::INV_PI * fmax_(SHADE_EPS, bs.wi.z) / bs.pdf * weight * ratio;
        out.dPa = v3(k1, k1, k1);
        out.dPr = scale(out.P, dlv * dadr);
      } else {  // k * spec with k = max(D(h) G / (4 wo.z pdfS), 0), pdfS = specularPdf(m)
        const V3 hv = hb;
        const float D = ggx_d(hv, a, a), G = ggx_g1(bs.wi, hv, a, a) * ggx_g1(si.wo, hv, a, a);
        const float k = fmax_(D * G / (4.0f * si.wo.z * bs.pdf), 0.0f);
        const float praw = ggx_d(m, a, a) * ggx_g1(si.wo, m, a, a) / (4.0f * si.wo.z);
        const float dlp = praw > SHADE_EPS ? dlog_ggx_d(m, a) + dlog_ggx_g1(si.wo, m, a) : 0.0f;
        const float dk =
            k > 0.0f ? k * (dlog_ggx_d(hv, a) + dlog_ggx_g1(bs.wi, hv, a) + dlog_ggx_g1(si.wo, hv, a) - dlp) : 0.0f;
        const float dw = env.enabled ? dph_dp0(bs.pdf, pe) * bs.pdf * dlp : 0.0f;
        const float dkw = ratio * (dlv * k * weight + dk * weight + k * dw) * dadr;
        const float ka = ratio * k * si.metallic * weight;
        out.dPa = v3(ka, ka, ka);
        out.dPr = v3(si.spec.x * dkw, si.spec.y * dkw, si.spec.z * dkw);
      }
    }
  }
  if (env.enabled) {
    const Sample es_ = sample_env(env, theta, h, si);
    if (dot(es_.wi, m) > 0.0f && es_.wi.z > 0.0f) {
      // createMaterialSampleRay (shade_hit.wgsl:339-348)
      const float lw = power_heuristic(es_.pdf, lambert_pdf(es_.wi));
      const V3 el = eval_lambert(si, es_);
      V3 scv = scale(v3((1.0f - f) * el.x, (1.0f - f) * el.y, (1.0f - f) * el.z), lw);
      const V3 hv = normalize(add(si.wo, es_.wi));
      const float p1 = specular_pdf(si, hv);
      const float sw = power_heuristic(es_.pdf, p1);
      const V3 ev = eval_specular(si, es_, hv);
      scv = add(scv, scale(v3(f * ev.x, f * ev.y, f * ev.z), sw));
      const V3 sdir = matvec(si.b1, si.b2, si.n, es_.wi);
      out.es = true;
      out.so = make_float4(si.origin.x, si.origin.y, si.origin.z, 0.0f);
      out.sd = make_float4(sdir.x, sdir.y, sdir.z, 0.0f);
      out.st = make_float4(scv.x * t4.x * ratio, scv.y * t4.y * ratio, scv.z * t4.z * ratio, t4.w);
      if (DERIV) {
        out.S = scale(scv, ratio);
        const float kl = (1.0f - f) * c::INV_PI * fmax_(SHADE_EPS, es_.wi.z) / es_.pdf * lw;
        const float D = ggx_d(hv, a, a), G1o = ggx_g1(si.wo, hv, a, a);
        const float ks = fmax_(D * ggx_g1(es_.wi, hv, a, a) * G1o / (4.0f * si.wo.z * es_.pdf), 0.0f);
        const float dlh = dlog_ggx_d(hv, a) + dlog_ggx_g1(si.wo, hv, a);
        const float dks = ks > 0.0f ? ks * (dlh + dlog_ggx_g1(es_.wi, hv, a)) : 0.0f;
        const float dp1 = D * G1o / (4.0f * si.wo.z) > SHADE_EPS ? p1 * dlh : 0.0f;
        const float dsw = -dph_dp0(p1, es_.pdf) * dp1;
        const float dsc = f * (dks * sw + ks * dsw);
        const float sa = ratio * (kl + f * ks * si.metallic * sw);
        out.dSa = v3(sa, sa, sa);
        out.dSr = v3(ratio * (dlv * scv.x + si.spec.x * dsc) * dadr, ratio * (dlv * scv.y + si.spec.y * dsc) * dadr,
                     ratio * (dlv * scv.z + si.spec.z * dsc) * dadr);
      }
    }
  }
}

// ---- the wavefront --------------------------------------------------------
// Paths are rendered a chunk at a time, all of a chunk's paths one bounce per
// round: closest hits (trace_lanes), shading, shadow rays (trace_lanes).  The
// random numbers of a vertex depend on pixel, sample and bounce only, so the
// queues need no order: blocks append rays as they come.  What a path adds to
// its pixel at each bounce is kept and summed afterwards in the order in which
// one thread per pixel would meet it (sample by sample, bounce by bounce), so
// the image has the same bits as a path-by-path loop.
//   A thread per pixel that walks its samples one after the other (the form
// before) kept 32 paths of different lengths in lockstep through traversal and
// shading: 0.8 Grays/s forward on the 512x512, 16 spp, 1.3M-triangle workload,
// where the same rays as queues run at the frame renderer's rate.
struct PathCount {  // one per chunk, zero at its start
  uint32_t rays[DIFF_MAX_DEPTH + 1], shadow[DIFF_MAX_DEPTH];
  uint32_t ticket[DIFF_MAX_DEPTH], shadow_ticket[DIFF_MAX_DEPTH];
};
struct PathTotal {
  unsigned long long rays;
  uint32_t err, pad;
};

// Buffers of a chunk of n paths.  Ray queues {origin, path}, {direction, -},
// {throughput, pixel}; per path the number of bounces it lived.
struct PathDev {
  float4 *o[2], *d[2], *t[2], *so, *sd, *st;
  uint4* hit;
  uint8_t* lived;
  float4* add;     // forward: [bounce][path] contribution
  float4* rec[6];  // adjoint: [bounce][path] vertex record
  uint32_t n;
  PathCount* count;
  PathTotal* total;
};

// A vertex record.  Its contribution is T S E, the next vertex's throughput
// T P; dPa / dSa: derivatives of P / S by the same channel of the albedo, dPr /
// dSr by the roughness; E: environment radiance, texel `tex` (-1: none).
//   0: T, material (-1: none, -2: not a vertex, an alpha pass-through)
//   1: P, dPa   2: dPr, dSa   3: S, -   4: dSr, tex   5: E, -
constexpr int REC_SKIP = -2;

struct ViewDev {
  CamState cam;
  float theta;
  uint32_t W, H;
  unsigned long long first;  // path index of the chunk's first path: sample * W * H + pixel
};

// Resident blocks of the closest-hit traversal (54 registers; 512x512, 16 spp,
// 1.3M triangles, forward and backward: 9 14.92 ms, 10 15.49, 8 15.5).
constexpr int PATH_TRACE_BLOCKS = 9;
constexpr int PATH_THREADS = 128;

__global__ void __launch_bounds__(PATH_THREADS) k_path_camera(PathDev D, ViewDev V, uint32_t sample_base) {
  __shared__ CamBasis s_basis;
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (threadIdx.x == 0) s_basis = camera_basis(V.cam);
  if (i == 0) D.count->rays[0] = D.n;
  __syncthreads();
  if (i >= D.n) return;
  const unsigned long long npix = (unsigned long long)V.W * V.H, p = V.first + i;
  const uint32_t pix = (uint32_t)(p % npix), px = pix % V.W, py = pix / V.W;
  V3 org, dir;
  camera_ray(V.cam, s_basis, px, py, V.W, V.H, (int32_t)(sample_base + (uint32_t)(p / npix)), org, dir);
  D.o[0][i] = make_float4(org.x, org.y, org.z, __uint_as_float(i));
  D.d[0][i] = make_float4(dir.x, dir.y, dir.z, 0.0f);
  D.t[0][i] = make_float4(1.0f, 1.0f, 1.0f, __uint_as_float(pix));
}

__global__ void __launch_bounds__(TRACE_THREADS, PATH_TRACE_BLOCKS) k_path_trace(SceneDev sc, PathDev D, int bounce) {
  __shared__ int sstack[LANES_SMEM][TRACE_THREADS];
  const int b = bounce & 1;
  trace_lanes<false, true>(
      sc, D.count->rays[bounce], D.count->ticket + bounce, &D.total->err, sstack,
      [&](uint32_t j, float4& o, float4& d) {
        o = D.o[b][j];
        d = D.d[b][j];
      },
      [&](uint32_t j, float, float, float, float t, int i, uint32_t bary) {
        __stcs(D.hit + j, make_uint4(__float_as_uint(t), (uint32_t)i, bary, 0u));
      });
}

// shade_miss.wgsl or shade_hit.wgsl for every ray of the bounce.
// (Resident blocks per SM: 512x512, 16 spp, 1.3M triangles, forward and backward:
// 6 14.77 ms, 7 14.74, 8 14.69, 9 14.66.  Sorting a tile's hits before its misses,
// so that one warp at most runs both branches, cost more in barriers and
// scattered accesses than it saved: 6 15.1, 8 14.9.)
constexpr int PATH_SHADE_BLOCKS = 8;
template <bool REC>
__global__ void __launch_bounds__(PATH_THREADS, PATH_SHADE_BLOCKS) k_path_shade(SceneDev sc, EnvDev env, DiffParams P,
                                                                                  PathDev D, ViewDev V, int bounce) {
  __shared__ uint32_t s_n[2], s_at[2];
  const uint32_t n = D.count->rays[bounce];
  const int b = bounce & 1;
  const unsigned long long npix = (unsigned long long)V.W * V.H;
  const uint32_t lane = threadIdx.x & 31u, ltmask = (1u << lane) - 1u;
  for (uint32_t base = blockIdx.x * PATH_THREADS; base < n; base += gridDim.x * PATH_THREADS) {
    const uint32_t j = base + threadIdx.x;
    if (threadIdx.x < 2) s_n[threadIdx.x] = 0;
    __syncthreads();
    bool next = false, es = false;
    float4 bo, bd, bt, so, sd, st;
    if (j < n) {
      const float4 o4 = __ldcs(D.o[b] + j), d4 = __ldcs(D.d[b] + j), t4 = __ldcs(D.t[b] + j);
      const uint4 hr = __ldcs(D.hit + j);
      const uint32_t path = __float_as_uint(o4.w);
      const size_t at = (size_t)bounce * D.n + path;
      D.lived[path] = (uint8_t)(bounce + 1);
      if ((int)hr.y < 0) {
        int tex;
        const V3 e = diff_env(P, V.theta, v3(d4.x, d4.y, d4.z), tex);
        if (REC) {
          D.rec[0][at] = make_float4(t4.x, t4.y, t4.z, __int_as_float(-1));
          D.rec[1][at] = make_float4(0.f, 0.f, 0.f, 0.f);
          D.rec[2][at] = make_float4(0.f, 0.f, 0.f, 0.f);
          D.rec[3][at] = make_float4(1.f, 1.f, 1.f, 0.f);
          D.rec[4][at] = make_float4(0.f, 0.f, 0.f, __int_as_float(tex));
          D.rec[5][at] = make_float4(e.x, e.y, e.z, 0.f);
        } else {
          D.add[at] = make_float4(e.x * t4.x, e.y * t4.y, e.z * t4.z, 0.0f);
        }
      } else {
        DiffShade s;
        const int32_t samples = (int32_t)(P.sample_base + (uint32_t)((V.first + path) / npix));
        shade_diff<REC>(sc, env, P, V.theta, samples, (uint32_t)bounce, o4, d4, t4, hr, s);
        next = s.eb && bounce + 1 < P.depth;
        es = s.es;
        bo = make_float4(s.bo.x, s.bo.y, s.bo.z, o4.w); bd = s.bd; bt = s.bt;
        so = make_float4(s.so.x, s.so.y, s.so.z, o4.w); sd = s.sd; st = s.st;
        if (REC) {
          if (s.pass && next) {  // changes nothing: not a vertex
            D.rec[0][at] = make_float4(0.f, 0.f, 0.f, __int_as_float(REC_SKIP));
          } else {
            const V3 zero = v3(0.0f, 0.0f, 0.0f);
            const V3 p = next ? s.P : zero, dpr = next ? s.dPr : zero;
            const float dpa = next ? s.dPa.x : 0.0f;
            const V3 q = s.emitted ? s.Qem : s.S;
            D.rec[0][at] = make_float4(t4.x, t4.y, t4.z, __int_as_float(s.emitted ? -1 : s.mat));
            D.rec[1][at] = make_float4(p.x, p.y, p.z, dpa);
            D.rec[2][at] = make_float4(dpr.x, dpr.y, dpr.z, s.emitted ? 0.0f : s.dSa.x);
            D.rec[3][at] = make_float4(q.x, q.y, q.z, 0.0f);
            D.rec[4][at] = make_float4(s.dSr.x, s.dSr.y, s.dSr.z, __int_as_float(-1));
            const float one = s.emitted ? 1.0f : 0.0f;  // a shadow ray that escapes writes its radiance
            D.rec[5][at] = make_float4(one, one, one, 0.0f);
          }
        } else {
          D.add[at] = s.emitted ? make_float4(s.em.x, s.em.y, s.em.z, 0.0f) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
    }
    // append: one counter update per block and queue
    const uint32_t mb = __ballot_sync(0xffffffffu, next), ms = __ballot_sync(0xffffffffu, es);
    uint32_t wb = 0, ws = 0;
    if (lane == 0) {
      if (mb) wb = atomicAdd(&s_n[0], (uint32_t)__popc(mb));
      if (ms) ws = atomicAdd(&s_n[1], (uint32_t)__popc(ms));
    }
    wb = __shfl_sync(0xffffffffu, wb, 0);
    ws = __shfl_sync(0xffffffffu, ws, 0);
    __syncthreads();
    if (threadIdx.x == 0 && s_n[0]) s_at[0] = atomicAdd(&D.count->rays[bounce + 1], s_n[0]);
    if (threadIdx.x == 32 && s_n[1]) s_at[1] = atomicAdd(&D.count->shadow[bounce], s_n[1]);
    __syncthreads();
    if (next) {
      const uint32_t k = s_at[0] + wb + (uint32_t)__popc(mb & ltmask);
      __stcs(D.o[b ^ 1] + k, bo);
      __stcs(D.d[b ^ 1] + k, bd);
      __stcs(D.t[b ^ 1] + k, bt);
    }
    if (es) {
      const uint32_t k = s_at[1] + ws + (uint32_t)__popc(ms & ltmask);
      __stcs(D.so + k, so);
      __stcs(D.sd + k, sd);
      __stcs(D.st + k, st);
    }
    __syncthreads();
  }
}

// trace_shadow.wgsl for the bounce's shadow rays; one that escapes adds the
// environment's radiance to its vertex (each vertex has at most one).
template <bool REC>
__global__ void __launch_bounds__(TRACE_THREADS, LANES_BLOCKS) k_path_shadow(SceneDev sc, DiffParams P, PathDev D,
                                                                             float theta, int bounce) {
  __shared__ int sstack[LANES_SMEM][TRACE_THREADS];
  trace_lanes<true, false>(
      sc, D.count->shadow[bounce], D.count->shadow_ticket + bounce, &D.total->err, sstack,
      [&](uint32_t j, float4& o, float4& d) {
        o = D.so[j];
        d = D.sd[j];
      },
      [&](uint32_t j, float dx, float dy, float dz, float, int i, uint32_t) {
        if (i >= 0) return;
        const size_t at = (size_t)bounce * D.n + __float_as_uint(D.so[j].w);
        int tex;
        const V3 e = diff_env(P, theta, v3(dx, dy, dz), tex);
        if (REC) {
          D.rec[4][at].w = __int_as_float(tex);
          D.rec[5][at] = make_float4(e.x, e.y, e.z, 0.0f);
        } else {
          const float4 st = D.st[j];
          float4 a = D.add[at];
          a.x += e.x * st.x;
          a.y += e.y * st.y;
          a.z += e.z * st.z;
          D.add[at] = a;
        }
      });
}

// Sums of the chunk's contributions, continuing image (the sums of the chunks
// before; `last`: then the mean).
__global__ void __launch_bounds__(PATH_THREADS) k_path_sum(PathDev D, unsigned long long first, uint32_t npix,
                                                           float4* __restrict__ image, float inv, int last) {
  const uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= npix) return;
  float4 acc = first ? image[pix] : make_float4(0.f, 0.f, 0.f, 0.f);
  const uint32_t r = (uint32_t)(first % npix);
  for (unsigned long long i = pix >= r ? pix - r : (unsigned long long)npix - r + pix; i < D.n; i += npix) {
    const int nb = D.lived[i];
    for (int b = 0; b < nb; b++) {
      const float4 c = __ldcs(D.add + (size_t)b * D.n + i);
      acc.x = acc.x + c.x;
      acc.y = acc.y + c.y;
      acc.z = acc.z + c.z;
    }
  }
  image[pix] = last ? make_float4(acc.x * inv, acc.y * inv, acc.z * inv, 0.0f) : acc;
}

// Sum of v over the lanes of `mask` holding the same key; the lowest such lane
// receives it (others get 0).  Every lane of `mask` must call it.
__device__ __forceinline__ float group_sum(unsigned peers, float v) {
  float sum = 0.0f;
  for (unsigned m = peers; m; m &= m - 1u) sum += __shfl_sync(peers, v, __ffs(m) - 1);
  return sum;
}

// The backward sweep of the chunk's paths: L_v = Q_v + P_v L_{v+1} from the last
// vertex, gradients per vertex.  Material terms: warp-aggregated atomics into
// per-block FP32 partials, flushed with FP64 atomics; environment terms:
// warp-aggregated per texel, added in FP64.
constexpr int SWEEP_THREADS = 256;
constexpr int SWEEP_PATHS = 8;  // paths per thread: the partials of a block cover 2048
__global__ void __launch_bounds__(SWEEP_THREADS) k_path_sweep(DiffParams P, PathDev D, unsigned long long first,
                                                              uint32_t npix, const float4* __restrict__ dimage,
                                                              double* __restrict__ g_albedo,
                                                              double* __restrict__ g_rough,
                                                              double* __restrict__ g_env) {
  extern __shared__ float spart[];  // n_mats x 4: albedo rgb, roughness
  for (uint32_t i = threadIdx.x; i < 4 * P.n_mats; i += blockDim.x) spart[i] = 0.0f;
  __syncthreads();
  const float inv = 1.0f / (float)P.spp;
  for (int q = 0; q < SWEEP_PATHS; q++) {
    const uint32_t i = (blockIdx.x * SWEEP_PATHS + q) * SWEEP_THREADS + threadIdx.x;
    float g[3] = {0.0f, 0.0f, 0.0f}, L[3] = {0.0f, 0.0f, 0.0f};
    int nv = 0;
    if (i < D.n) {
      const float4 dv = dimage[(uint32_t)((first + i) % npix)];
      g[0] = dv.x * inv; g[1] = dv.y * inv; g[2] = dv.z * inv;
      nv = D.lived[i];
    }
    const int most = __reduce_max_sync(0xffffffffu, nv);
    for (int v = most - 1; v >= 0; v--) {
      int mkey = -1, tkey = -1;
      float da[3] = {0.f, 0.f, 0.f}, dr = 0.0f, de[3] = {0.f, 0.f, 0.f};
      if (v < nv) {
        const size_t at = (size_t)v * D.n + i;
        const float4 r0 = __ldcs(D.rec[0] + at);
        if (__float_as_int(r0.w) != REC_SKIP) {
          const float4 r1 = __ldcs(D.rec[1] + at), r2 = __ldcs(D.rec[2] + at), r3 = __ldcs(D.rec[3] + at),
                       r4 = __ldcs(D.rec[4] + at), r5 = __ldcs(D.rec[5] + at);
          mkey = __float_as_int(r0.w);
          tkey = __float_as_int(r4.w);
          const float T[3] = {r0.x, r0.y, r0.z}, Pv[3] = {r1.x, r1.y, r1.z}, dPr[3] = {r2.x, r2.y, r2.z},
                      S[3] = {r3.x, r3.y, r3.z}, dSr[3] = {r4.x, r4.y, r4.z}, E[3] = {r5.x, r5.y, r5.z};
#pragma unroll
          for (int c = 0; c < 3; c++) {
            const float gt = g[c] * T[c];
            da[c] = gt * (r2.w * E[c] + r1.w * L[c]);
            dr += gt * (dSr[c] * E[c] + dPr[c] * L[c]);
            de[c] = gt * S[c];
            L[c] = S[c] * E[c] + Pv[c] * L[c];
          }
        }
      }
      const uint32_t lane = threadIdx.x & 31u;
      const unsigned mp = __match_any_sync(0xffffffffu, mkey);
      if (mkey >= 0) {
        const float s0 = group_sum(mp, da[0]), s1 = group_sum(mp, da[1]), s2 = group_sum(mp, da[2]),
                    s3 = group_sum(mp, dr);
        if ((int)lane == __ffs(mp) - 1) {
          atomicAdd(&spart[4 * mkey + 0], s0);
          atomicAdd(&spart[4 * mkey + 1], s1);
          atomicAdd(&spart[4 * mkey + 2], s2);
          atomicAdd(&spart[4 * mkey + 3], s3);
        }
      }
      __syncwarp();
      const unsigned tp = __match_any_sync(0xffffffffu, tkey);
      if (tkey >= 0) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const float se = group_sum(tp, de[c]);
          if ((int)lane == __ffs(tp) - 1 && se != 0.0f) atomicAdd(g_env + 3 * (size_t)tkey + c, (double)se);
        }
      }
      __syncwarp();
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < 4 * P.n_mats; i += blockDim.x) {
    const float v = spart[i];
    if (v != 0.0f) {
      if ((i & 3u) == 3u) atomicAdd(g_rough + (i >> 2), (double)v);
      else atomicAdd(g_albedo + 3 * (i >> 2) + (i & 3u), (double)v);
    }
  }
}

// After a chunk: its rays.  After the last: status and ray count for the host.
__global__ void k_path_end(PathCount* c, PathTotal* t, int depth, uint32_t* host) {
  unsigned long long r = t->rays;
  for (int b = 0; b < depth; b++) r += (unsigned long long)c->rays[b] + c->shadow[b];
  t->rays = r;
  host[0] = t->err;
  host[1] = (uint32_t)(r & 0xffffffffu);
  host[2] = (uint32_t)(r >> 32);
}

namespace {

int diff_fail(pk_ctx* c, int code, const char* msg) {
  c->err = msg;
  return code;
}

int diff_check(pk_ctx* c, const pk_diff_params* p, DiffParams& dp) {
  if (const char* gap = c->scene_gap()) return diff_fail(c, PK_ERR_STATE, gap);
  if (!c->W || !c->H) return diff_fail(c, PK_ERR_STATE, "pk_diff: call pk_configure first");
  if (!c->cam_set) return diff_fail(c, PK_ERR_STATE, "pk_diff: call pk_set_camera first");
  if (!c->diff_env_ready) return diff_fail(c, PK_ERR_STATE, "pk_diff: call pk_diff_set_env_sampling first");
  if (!p || !p->albedo3 || !p->roughness || !p->metallic || !p->env_rgb)
    return diff_fail(c, PK_ERR_ARG, "pk_diff: null argument");
  if (p->n_mats < c->n_mats || p->n_mats == 0 || p->n_mats > 4096)
    return diff_fail(c, PK_ERR_ARG, "pk_diff: n_mats must cover the scene's materials (at most 4096)");
  if (p->env_w != c->diff_env_w || p->env_h != c->diff_env_h)
    return diff_fail(c, PK_ERR_ARG, "pk_diff: env size differs from the sampling tables' (pk_diff_set_env_sampling)");
  if (!p->spp || p->spp > 65536 || p->depth < 1 || p->depth > DIFF_MAX_DEPTH)
    return diff_fail(c, PK_ERR_ARG, "pk_diff: bad spp or depth (1..8)");
  dp = DiffParams{p->albedo3, p->roughness, p->roughness_sampling ? p->roughness_sampling : p->roughness,
                  p->metallic, p->n_mats, p->env_rgb, (int)p->env_w, (int)p->env_h, (int)p->spp, (int)p->depth,
                  p->sample_base};
  return PK_OK;
}

EnvDev diff_env_dev(pk_ctx* c) {
  return EnvDev{nullptr, c->diff_bins.p, c->diff_coords.p, c->diff_pdf.p, (int)c->diff_env_w, (int)c->diff_env_h,
                (int)c->diff_env_nb, 1, nullptr};
}

// Paths per chunk: enough to fill the GPU many times over (the tail of a
// bounce's longest rays costs as much as some 10^5 rays), within PATH_SPACE
// bytes of workspace that the context keeps; half as many, again and again, when
// the device has no memory for them, down to PATH_LEAST (1 MB at the most).
constexpr unsigned long long PATH_CHUNK = 1ull << 22;
constexpr unsigned long long PATH_SPACE = 3ull << 30;
constexpr unsigned long long PATH_LEAST = 1ull << 10;

// Renders every path (REC: recording vertices) chunk by chunk; after(D, first,
// last) turns a chunk into its part of the result.
template <bool REC, class F>
int run_paths(pk_ctx* c, const char* what, const DiffParams& P, F after) {
  const cudaStream_t st = c->stream;
  const uint32_t npix = c->W * c->H;
  const unsigned long long total = (unsigned long long)npix * (unsigned long long)P.spp;
  const unsigned long long per = 9 * 16 + 16 + 4 + (unsigned long long)P.depth * 16 * (REC ? 6 : 1);
  unsigned long long chunk = std::min(std::min(total, PATH_CHUNK), PATH_SPACE / per);
  const size_t head = 512;
  static_assert(sizeof(PathCount) + sizeof(PathTotal) <= 512, "header");
  for (;; chunk = (chunk + 1) / 2) {
    const size_t need = head + (size_t)(chunk * per) + 64;
    if (c->diff_space.cap >= need) break;
    try {
      c->diff_space.alloc(need);  // grows, at most to PATH_SPACE; goes with the context
      break;
    } catch (CudaError&) {
      if (chunk <= PATH_LEAST) throw;
    }
  }
  const size_t n = (size_t)chunk;
  unsigned char* at = c->diff_space.p;
  auto take = [&](size_t bytes) {
    unsigned char* p = at;
    at += (bytes + 15) / 16 * 16;
    return p;
  };
  PathDev D{};
  D.total = reinterpret_cast<PathTotal*>(at);
  D.count = reinterpret_cast<PathCount*>(at + sizeof(PathTotal));
  at += head;
  for (int b = 0; b < 2; b++) {
    D.o[b] = reinterpret_cast<float4*>(take(16 * n));
    D.d[b] = reinterpret_cast<float4*>(take(16 * n));
    D.t[b] = reinterpret_cast<float4*>(take(16 * n));
  }
  D.so = reinterpret_cast<float4*>(take(16 * n));
  D.sd = reinterpret_cast<float4*>(take(16 * n));
  D.st = reinterpret_cast<float4*>(take(16 * n));
  D.hit = reinterpret_cast<uint4*>(take(16 * n));
  if (REC)
    for (int k = 0; k < 6; k++) D.rec[k] = reinterpret_cast<float4*>(take(16 * n * (size_t)P.depth));
  else
    D.add = reinterpret_cast<float4*>(take(16 * n * (size_t)P.depth));
  D.lived = take(n);
  const SceneDev sc = c->dropin_scene();
  const EnvDev env = diff_env_dev(c);
  check(cudaMemsetAsync(D.total, 0, sizeof(PathTotal), st), "memset");
  for (unsigned long long first = 0; first < total; first += chunk) {
    D.n = (uint32_t)std::min(chunk, total - first);
    const bool last = first + chunk >= total;
    const ViewDev V{c->cam_host, c->theta_next, c->W, c->H, first};
    check(cudaMemsetAsync(D.count, 0, sizeof(PathCount), st), "memset");
    const unsigned blocks = (D.n + PATH_THREADS - 1) / PATH_THREADS;
    const unsigned lanes = std::min((unsigned)c->sms * LANES_BLOCKS, blocks);
    const unsigned shade = std::min((unsigned)c->sms * 4 * PATH_SHADE_BLOCKS, blocks);
    k_path_camera<<<blocks, PATH_THREADS, 0, st>>>(D, V, P.sample_base);
    for (int b = 0; b < P.depth; b++) {
      k_path_trace<<<lanes, TRACE_THREADS, 0, st>>>(sc, D, b);
      k_path_shade<REC><<<shade, PATH_THREADS, 0, st>>>(sc, env, P, D, V, b);
      k_path_shadow<REC><<<lanes, TRACE_THREADS, 0, st>>>(sc, P, D, V.theta, b);
    }
    after(D, first, last);
    k_path_end<<<1, 1, 0, st>>>(D.count, D.total, P.depth, c->host_words_dev);
    check(cudaGetLastError(), what);
  }
  check(cudaStreamSynchronize(st), "sync");
  const volatile uint32_t* h = c->host_words;
  c->diff_rays = (unsigned long long)h[1] | ((unsigned long long)h[2] << 32);
  if (h[0]) {
    c->err = std::string(what) + ": device error flags (traversal stack)";
    return PK_ERR_DEVICE;
  }
  return PK_OK;
}

}  // namespace
}  // namespace pk

using namespace pk;

extern "C" int pk_diff_set_env_sampling(pk_ctx* c, const float* env_rgb, uint32_t w, uint32_t h) {
  if (!c) return PK_ERR_ARG;
  try {
    check(cudaSetDevice(c->device), "cudaSetDevice");
    if (!env_rgb || !w || !h || (uint64_t)w * h > (1ull << 26))
      return diff_fail(c, PK_ERR_ARG, "pk_diff_set_env_sampling: null map or bad size");
    std::string why;
    uint32_t nb = 0;
    c->diff_env_ready = false;
    if (build_env_tables_gpu_f32(c->scratch(), env_rgb, w, h, c->diff_bins, nb, c->diff_coords, c->diff_pdf, why)) {
      c->err = "pk_diff_set_env_sampling: " + why;
      return PK_ERR_ARG;
    }
    c->diff_env_w = w;
    c->diff_env_h = h;
    c->diff_env_nb = nb;
    c->diff_env_ready = true;
    return PK_OK;
  } catch (CudaError& e) {
    c->err = e.what();
    return PK_ERR_CUDA;
  }
}

extern "C" int pk_diff_env_info(pk_ctx* c, uint32_t* w, uint32_t* h, uint32_t* nb) {
  if (!c || !w || !h || !nb) return PK_ERR_ARG;
  if (!c->diff_env_ready) return diff_fail(c, PK_ERR_STATE, "pk_diff_env_info: no sampling tables");
  *w = c->diff_env_w;
  *h = c->diff_env_h;
  *nb = c->diff_env_nb;
  return PK_OK;
}

extern "C" int pk_diff_env_download(pk_ctx* c, int32_t* bins2, int32_t* coords2, float* pdf) {
  if (!c || !bins2 || !coords2 || !pdf) return PK_ERR_ARG;
  if (!c->diff_env_ready) return diff_fail(c, PK_ERR_STATE, "pk_diff_env_download: no sampling tables");
  try {
    check(cudaSetDevice(c->device), "cudaSetDevice");
    const size_t n = (size_t)c->diff_env_w * c->diff_env_h;
    check(cudaMemcpyAsync(bins2, c->diff_bins.p, 8 * (size_t)c->diff_env_nb, cudaMemcpyDeviceToHost, c->stream), "D2H");
    check(cudaMemcpyAsync(coords2, c->diff_coords.p, 8 * n, cudaMemcpyDeviceToHost, c->stream), "D2H");
    check(cudaMemcpyAsync(pdf, c->diff_pdf.p, 4 * n, cudaMemcpyDeviceToHost, c->stream), "D2H");
    check(cudaStreamSynchronize(c->stream), "sync");
    return PK_OK;
  } catch (CudaError& e) {
    c->err = e.what();
    return PK_ERR_CUDA;
  }
}

extern "C" int pk_diff_render(pk_ctx* c, const pk_diff_params* p, float* image4) {
  if (!c) return PK_ERR_ARG;
  try {
    check(cudaSetDevice(c->device), "cudaSetDevice");
    DiffParams dp;
    const int rc = diff_check(c, p, dp);
    if (rc != PK_OK) return rc;
    if (!image4) return diff_fail(c, PK_ERR_ARG, "pk_diff_render: null image");
    const uint32_t npix = c->W * c->H;
    float4* image = reinterpret_cast<float4*>(image4);
    const float inv = 1.0f / (float)dp.spp;
    return run_paths<false>(c, "pk_diff_render", dp, [&](const PathDev& D, unsigned long long first, bool last) {
      k_path_sum<<<(npix + PATH_THREADS - 1) / PATH_THREADS, PATH_THREADS, 0, c->stream>>>(D, first, npix, image, inv,
                                                                                           last ? 1 : 0);
    });
  } catch (CudaError& e) {
    c->err = e.what();
    return PK_ERR_CUDA;
  }
}

extern "C" int pk_diff_backward(pk_ctx* c, const pk_diff_params* p, const float* d_image4, double* g_albedo3,
                                double* g_roughness, double* g_env_rgb) {
  if (!c) return PK_ERR_ARG;
  try {
    check(cudaSetDevice(c->device), "cudaSetDevice");
    DiffParams dp;
    const int rc = diff_check(c, p, dp);
    if (rc != PK_OK) return rc;
    if (!d_image4 || !g_albedo3 || !g_roughness || !g_env_rgb)
      return diff_fail(c, PK_ERR_ARG, "pk_diff_backward: null buffer");
    const uint32_t npix = c->W * c->H;
    const size_t smem = 16 * (size_t)p->n_mats;
    if (smem > 48 * 1024)
      check(cudaFuncSetAttribute(k_path_sweep, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "attr");
    return run_paths<true>(c, "pk_diff_backward", dp, [&](const PathDev& D, unsigned long long first, bool) {
      const unsigned per = SWEEP_THREADS * SWEEP_PATHS;
      k_path_sweep<<<(D.n + per - 1) / per, SWEEP_THREADS, smem, c->stream>>>(
          dp, D, first, npix, reinterpret_cast<const float4*>(d_image4), g_albedo3, g_roughness, g_env_rgb);
    });
  } catch (CudaError& e) {
    c->err = e.what();
    return PK_ERR_CUDA;
  }
}

extern "C" int pk_diff_rays(pk_ctx* c, unsigned long long* rays) {
  if (!c || !rays) return PK_ERR_ARG;
  *rays = c->diff_rays;
  return PK_OK;
}
