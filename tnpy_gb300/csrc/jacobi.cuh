// Rotation angles of the Jacobi eigensolvers.
#pragma once

#include <cuda_runtime.h>

namespace tnx {
namespace jac {

// round-robin (circle method) pair k of round r for np (even) players, p < q
__device__ __forceinline__ void pair_of(int k, int r, int np, int& p, int& q) {
  const int m1 = np - 1;
  p = k - 1 + r;
  q = np - 2 - k + r;
  p = k == 0 ? 0 : 1 + (p >= m1 ? p - m1 : p);
  q = 1 + (q >= m1 ? q - m1 : q);
  if (p > q) {
    const int t = p;
    p = q;
    q = t;
  }
}

// double <-> float by integer operations (the conversions run on the FP64 pipe): truncated to 24
// bits, zero below 2^-126; |x| < 2^127
__device__ __forceinline__ float to_float(double x) {
  const unsigned hi = unsigned(__double2hiint(x)), lo = unsigned(__double2loint(x));
  const int e = int((hi >> 20) & 0x7ffu) - 896;
  return e <= 0 ? 0.f : __uint_as_float((hi & 0x80000000u) | (unsigned(e) << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29));
}
__device__ __forceinline__ double to_double(float x) {
  const unsigned u = __float_as_uint(x), m = u & 0x7fffffffu;
  if (m < 0x00800000u) return 0.0;
  return __hiloint2double(int((u & 0x80000000u) | ((m >> 3) + (896u << 20))), int(m << 29));
}
// x 2^-e for |x| 2^-e < 2^1023; zero where it would be subnormal
__device__ __forceinline__ double scale_exp(double x, int e) {
  const int hi = __double2hiint(x), ex = ((hi >> 20) & 0x7ff) - e;
  return ex <= 0 ? 0.0 : __hiloint2double(hi - (e << 20), __double2loint(x));
}

// +-0 gives 0
__device__ __forceinline__ unsigned long long bits(double x) {
  return static_cast<unsigned long long>(__double_as_longlong(x)) << 1;
}
__device__ __forceinline__ unsigned long long bits(float x) {
  return __float_as_uint(x) << 1;
}

// integer in the order of x, +-0 equal; NaN beyond the infinities, so that ranks by it are always a permutation
__device__ __forceinline__ long long sort_key(double x) {
  const long long k = bits(x) == 0 ? 0 : __double_as_longlong(x);
  return k < 0 ? k ^ 0x7fffffffffffffffLL : k;
}
__device__ __forceinline__ int sort_key(float x) {
  const int k = bits(x) == 0 ? 0 : __float_as_int(x);
  return k < 0 ? k ^ 0x7fffffff : k;
}

// 1 / sqrt(d) for d in FP32's normal range: FP32 seed and one third-order step (error 2^-66 before
// the last rounding), five FP64 instructions
__device__ __forceinline__ double rsqrt_exact(double d) {
  const double y = to_double(rsqrtf(to_float(d))), r = fma(-d, y * y, 1.0);
  return fma(y * r, fma(0.375, r, 0.5), y);
}

// Rotation that zeroes a_pq: t = tan, c, s with |t| <= 1; d = a_qq - a_pp (d = 0: t = 1). FP64
// instructions hold the pipe for 64 clocks a warp, so the tangent comes from FP32 (approximate
// reciprocal and root, exponents aligned by integer arithmetic) and two corrections against
// a_pq t^2 + d t - a_pq = 0, and c = 1 / sqrt(1 + t^2) from an FP32 seed by one third-order step.
__device__ __forceinline__ void angle(double apq, double d, double& t, double& c, double& s) {
  const int ea = (__double2hiint(apq) >> 20) & 0x7ff, ed = (__double2hiint(d) >> 20) & 0x7ff;
  const int e = max(ea, ed) - 1023;  // both below 2 after the scaling, the larger one above 1
  const double a1 = scale_exp(apq, e), d1 = scale_exp(d, e);
  const float af = to_float(a1), df = to_float(d1), a2 = 2.f * af;
  float tf = 1.f;
  double tt = 1.0;
  if (ed - ea > 30) {
    // t = a_pq / d to FP64 accuracy (the next term is (a_pq / d)^2 < 2^-60 of it), by an FP32 seed of
    // 1 / d and one third-order step: a_pq itself may lie far below FP32's range here
    const double z = to_double(__fdividef(1.f, df)), r = fma(-d1, z, 1.0);
    tt = a1 * fma(z * r, 1.0 + r, z);
    tf = 0.f;
  } else if (bits(d1) != 0) {
    const float h = fmaf(df, df, a2 * a2);
    const unsigned sign = unsigned(__double2hiint(d1)) & 0x80000000u;
    tf = __uint_as_float(sign | 0x3f800000u) * __fdividef(a2, fmaf(h, rsqrtf(h), fabsf(df)));
    // corrections against f(t) = a_pq t^2 + d t - a_pq, f' = 2 a_pq t + d
    const float inv = __fdividef(1.f, fmaf(a2, tf, df));
    tt = to_double(tf);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const double f = fma(fma(a1, tt, d1), tt, -a1);
      tt -= to_double(to_float(f) * inv);
    }
  }
  const double y = to_double(rsqrtf(fmaf(tf, tf, 1.f)));
  const double r = fma(-fma(tt, tt, 1.0), y * y, 1.0);  // 1 - (1 + t^2) y^2
  c = fma(y * r, fma(0.375, r, 0.5), y);
  s = tt * c;
  t = tt;
}
// the same in FP32; |d| / |apq| < 1e9
__device__ __forceinline__ void angle(float apq, float d, float& t, float& c, float& s) {
  const float th = d / (2.f * apq);
  t = (th >= 0.f ? 1.f : -1.f) / (fabsf(th) + sqrtf(fmaf(th, th, 1.f)));
  c = 1.f / sqrtf(fmaf(t, t, 1.f));
  s = t * c;
}

}  // namespace jac
}  // namespace tnx
