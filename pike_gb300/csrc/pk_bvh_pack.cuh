// pk_bvh_pack.cuh -- trace_pass.js's normaliser and node quantisation, shared by
// the BVH builders.
#pragma once
#include <cuda_runtime.h>
#include <cmath>
#include <cstdint>

namespace pk {

struct Norm {
  double c[3], scale;  // centre, 2 / longest
};
// #makeNormalizer (trace_pass.js:202-211) of the root box, in double, JavaScript order.
inline double norm_js_max(double a, double b) {
  return (a != a || b != b) ? NAN : (a > b ? a : (b > a ? b : (std::signbit(a) ? b : a)));
}
inline Norm make_norm(const double mn[3], const double mx[3]) {
  Norm n;
  double span[3];
  for (int i = 0; i < 3; i++) {
    span[i] = mx[i] - mn[i];
    n.c[i] = mn[i] + span[i] * 0.5;
  }
  n.scale = 2.0 / norm_js_max(norm_js_max(span[0], span[1]), span[2]);
  return n;
}

// ECMAScript ToInt16: truncate, wrap modulo 2^16; non-finite -> 0.  Normalised
// bounds are within 32768 in magnitude, where the low 16 bits of the truncated
// value are the answer; fmod serves the rest.
__device__ __forceinline__ int js_toint16(double v) {
  if (fabs(v) < 2147483000.0) return (int)(int16_t)(uint16_t)((uint32_t)(int)v & 0xffffu);
  if (!isfinite(v)) return 0;
  double m = fmod(trunc(v), 65536.0);
  if (m < 0.0) m += 65536.0;
  int mi = (int)m;
  if (mi >= 32768) mi -= 65536;
  return mi;
}
// trace_pass.js:213-218 quantizeVec2ToInt on the normalised {max, min} of an axis.
__device__ __forceinline__ int32_t quantize_bounds(const Norm& n, int a, double mn, double mx) {
  const double hi = (mx - n.c[a]) * n.scale, lo = (mn - n.c[a]) * n.scale;
  const int s0 = js_toint16(hi * (hi > 0.0 ? 32767.0 : 32768.0));
  const int s1 = js_toint16(lo * (lo > 0.0 ? 32767.0 : 32768.0));
  return (int32_t)((uint32_t)(uint16_t)s0 | ((uint32_t)(uint16_t)s1 << 16));
}

void launch_norm_verts(cudaStream_t s, const double* pos3, uint32_t n, const Norm& norm, float4* verts4);

}  // namespace pk
