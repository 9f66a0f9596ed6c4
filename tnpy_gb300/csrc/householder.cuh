// Scalars of a Householder reflector in FP64.
#pragma once

#include <cuda_runtime.h>

#include "jacobi.cuh"

namespace tnx {

// Column with pivot alpha and sigma = sum of squares below it: beta = -sign(alpha) |x| takes the pivot's
// place, v = scale x below it (v = 1 at it), H = I - tau v v^T; the identity where sigma is zero.
// The root and the reciprocal come from FP32 seeds and third-order steps on exponents scaled to [1, 4):
// 20 FP64 instructions of 64 clocks each in the one warp that the others wait for, where sqrt and two
// divisions are over 60.
__device__ __forceinline__ void reflector(double alpha, double sigma, double& beta, double& tau, double& scale) {
  tau = scale = 0.0;
  beta = alpha;
  if (jac::bits(sigma) == 0) return;
  const double t2 = fma(alpha, alpha, sigma);
  const int ex = (__double2hiint(t2) >> 20) & 0x7ff;
  if (ex == 2047 || ex == 0) {  // Inf, NaN or a subnormal square
    const double nrm = sqrt(t2);
    beta = alpha >= 0.0 ? -nrm : nrm;
    tau = (beta - alpha) / beta;
    scale = 1.0 / (alpha - beta);
    return;
  }
  // t2 = s 2^e with even e and s in [1, 4): nrm = s y, y = 1 / sqrt(s)
  const int e = (ex - 1023) & ~1, h = e / 2;
  const double s = jac::scale_exp(t2, e), y = jac::rsqrt_exact(s), a = jac::scale_exp(fabs(alpha), h);
  double nrm = s * y;
  nrm = fma(0.5 * y, fma(-nrm, nrm, s), nrm);  // correctly rounded but for rare ties
  tau = fma(a, y, 1.0);
  // 1 / (|alpha| + nrm): FP32 seed, one third-order step
  const double d = a + nrm, z = jac::to_double(__fdividef(1.f, jac::to_float(d))), r = fma(-d, z, 1.0);
  const double inv = jac::scale_exp(fma(z * r, 1.0 + r, z), h);
  nrm = jac::scale_exp(nrm, -h);
  const bool neg = __double2hiint(alpha) < 0 && jac::bits(alpha) != 0;
  beta = neg ? nrm : -nrm;
  scale = neg ? -inv : inv;
}

}  // namespace tnx
