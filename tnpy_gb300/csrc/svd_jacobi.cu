// Singular value decomposition by one-sided (Hestenes) Jacobi in FP64, replacing
// np.linalg.svd in linalg.svd (tnpy/linalg.py:9-23) and the Schmidt values of the SVD gauge
// move (tnpy/matrix_product_state.py:200-223) where they are reported.
//
// The columns of a working copy C of A (m x n, m >= n) are rotated in pairs until every pair is
// orthogonal to working accuracy: for columns (p, q) with a = |c_p|^2, b = |c_q|^2, g = c_p.c_q,
// the plane rotation that zeroes g is applied to C and to V (V starts as the identity), so that
// C = A V keeps orthogonal columns at the end: sigma_j = |c_j|, u_j = c_j / sigma_j, A = U S V^T.
// The singular values come from the matrix itself, not from a Gram matrix A^T A, so a small
// sigma keeps an absolute error of ~eps * sigma_max instead of ~sqrt(eps) * sigma_max.
//
// Parallel order: the round-robin ("circle") tournament on ne = n rounded up to even columns
// (a zero column pads odd n): each of the ne - 1 rounds rotates ne / 2 disjoint pairs, one CTA
// per pair; a sweep is ne - 1 launches, and sweeps repeat until a sweep rotates no pair
// (|g| <= tol sqrt(a b), tol = sqrt(m) * 2^-52) or 40 sweeps pass. The host reads one counter
// and one mark per sweep. Working copies are column-major so that every column is contiguous.
//
// What bounds it: the chain of one pair, an FP64 instruction holding its sub-partition's pipe for 64
// clocks a warp, and the launches. A pair takes four warps (eight above 1024 rows), one to each
// sub-partition; the three dot products are reduced together (six additions a warp instead of
// fifteen) and the warps' sums by one lane per value; every warp computes the angle itself (jac::angle,
// 17 FP64 instructions, with an FP32 test for orthogonality on aligned exponents). The next round's
// launch overlaps the end of this one (programmatic dependent launch). m = n = 128: 2.9 us a round, 8 us
// with eight warps, one thread's serial sums, exact roots and divisions; singular values of a
// 1024 x 1024 R 295 -> 105 ms, with vectors 337 -> 243 ms.
//
// Singular values alone of a square matrix may come from its transpose: where the mass lies above
// the diagonal, as in the R of a QR, the columns of A^T are far closer to orthogonal (the 128 x 128 R
// of a middle bond takes 7 sweeps instead of 23).
#include <cuda_runtime.h>

#include <cmath>

#include "jacobi.cuh"
#include "tnx_internal.cuh"

namespace tnx {
namespace {

constexpr int JT = 256;
constexpr int kMaxSweeps = 40;

// C = A column by column (or A^T, square A, where flip[0] is set), V = I
__global__ void jac_init_kernel(const double* __restrict__ A, int64_t m, int64_t n, int64_t ne,
                                double* __restrict__ C, double* __restrict__ V, const int* __restrict__ flip) {
  const int64_t total = m * ne;
  const bool tr = flip && flip[0];
  for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < total; e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t j = e / m, i = e - j * m;
    C[e] = j < n ? A[tr ? j * n + i : i * n + j] : 0.0;
  }
  if (V) {
    const int64_t tv = ne * ne;
    for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < tv; e += int64_t(gridDim.x) * blockDim.x)
      V[e] = (e / ne == e % ne) ? 1.0 : 0.0;
  }
}

__device__ __forceinline__ void pair_of(int round, int k, int ne, int& p, int& q) {
  if (k == 0) {
    p = ne - 1;
    q = round;
  } else {
    p = (round + k) % (ne - 1);
    q = (round - k + (ne - 1)) % (ne - 1);
  }
}

// Sums over the CTA of the threads' a, b and g: in lane l of every warp, that of a (l mod 4 = 0), g (1 and 3) or b (2)
template <int WARPS>
__device__ __forceinline__ double pair_sums(double a, double b, double g, double (&red)[WARPS][4]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  // lanes 0-15 go on with a, 16-31 with b, then every other eight of them with g
  const bool hi = lane & 16, mid = lane & 8;
  double x = hi ? b : a;
  const double give = hi ? a : b;
  x += __shfl_xor_sync(0xffffffffu, give, 16);
  g += __shfl_xor_sync(0xffffffffu, g, 16);
  double z = mid ? g : x;
  const double give2 = mid ? x : g;
  z += __shfl_xor_sync(0xffffffffu, give2, 8);
  for (int o = 4; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
  if ((lane & 7) == 0) red[w][lane >> 3] = z;  // 0: a, 1 and 3: g, 2: b
  __syncthreads();
  double sum = red[0][lane & 3];
#pragma unroll
  for (int i = 1; i < WARPS; ++i) sum += red[i][lane & 3];
  return sum;
}
__device__ __forceinline__ void pair_share(double sum, double& a, double& b, double& g) {
  a = __shfl_sync(0xffffffffu, sum, 0);
  g = __shfl_sync(0xffffffffu, sum, 1);
  b = __shfl_sync(0xffffffffu, sum, 2);
}

// x <- c x - s y, y <- s x + c y
template <int T>
__device__ __forceinline__ void turn(double* xs, double* ys, int64_t n, double c, double s) {
#pragma unroll 4
  for (int64_t i = threadIdx.x; i < n; i += T) {
    const double x = xs[i], y = ys[i];
    xs[i] = fma(c, x, -s * y);
    ys[i] = fma(s, x, c * y);
  }
}

// A squared norm below 2^-TINY_EXP: their product with the tolerance may leave the normal range, and the sums may have
// lost bits to it. Where neither column is longer than 2^-150 the sums are taken again of the columns times 2^600
// (the angle does not change); otherwise g is well inside the range. FP64 roots and divisions: a rare case, in an
// instantiation of its own (47 registers against 32) that takes over once a sweep has met such a pair.
constexpr int TINY_EXP = 800;
template <int WARPS>
__device__ __forceinline__ void tiny_pair(double a, double b, double g, double* cp, double* cq, int64_t m, double* vp,
                                       double* vq, int ne, float tol, int* rotated, double (&red)[WARPS][4]) {
  constexpr int T = 32 * WARPS;
  if (fmax(a, b) < 0x1p-300) {
    a = b = g = 0.0;
    for (int64_t i = threadIdx.x; i < m; i += T) {
      const double x = cp[i] * 0x1p600, y = cq[i] * 0x1p600;
      a = fma(x, x, a);
      b = fma(y, y, b);
      g = fma(x, y, g);
    }
    __syncthreads();  // red has been read by all
    pair_share(pair_sums<WARPS>(a, b, g, red), a, b, g);
  }
  if (!(fabs(g) > double(tol) * sqrt(a) * sqrt(b))) return;
  // t = tan(theta): the smaller root of t^2 + 2 zeta t - 1 = 0, zeta = (b - a) / (2 g)
  const double zeta = (b - a) / (2.0 * g), az = fabs(zeta);
  const double t = copysign(az > 1e100 ? 0.5 / az : 1.0 / (az + sqrt(fma(zeta, zeta, 1.0))), zeta);
  const double c = 1.0 / sqrt(fma(t, t, 1.0)), s = c * t;
  if (jac::bits(s) == 0) return;
  if (threadIdx.x == 0) atomicAdd(rotated, 1);
  turn<T>(cp, cq, m, c, s);
  if (vp) turn<T>(vp, vq, ne, c, s);
}

// rotated[0]: rotations of the sweep; rotated[TINY_AT]: set where a pair was left to the form with TINY
constexpr int TINY_AT = 2;
template <int WARPS, bool TINY>
__global__ void __launch_bounds__(32 * WARPS) jac_round_kernel(double* __restrict__ C, int64_t m,
                                                              double* __restrict__ V, int ne, int round, float tol,
                                                              int* __restrict__ rotated) {
  constexpr int T = 32 * WARPS;
  __shared__ double red[WARPS][4];
  int p, q;
  pair_of(round, blockIdx.x, ne, p, q);
  double* cp = C + int64_t(p) * m;
  double* cq = C + int64_t(q) * m;
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the round before has written the columns
  double a = 0.0, b = 0.0, g = 0.0;
#pragma unroll 4
  for (int64_t i = threadIdx.x; i < m; i += T) {
    const double x = cp[i], y = cq[i];
    a = fma(x, x, a);
    b = fma(y, y, b);
    g = fma(x, y, g);
  }
  const double sum = pair_sums<WARPS>(a, b, g, red);
  // the next round's CTAs come in now and wait; triggered any earlier, several rounds of them pile up
  // (1024 columns: 330 against 105 ms)
  asm volatile("griddepcontrol.launch_dependents;");
  pair_share(sum, a, b, g);
  // |g| > tol sqrt(a b) in FP32, a and b scaled into [1, 4) by even powers of two and g to match; a
  // squared norm of zero has no direction to rotate
  const int xa = (__double2hiint(a) >> 20) & 0x7ff, xb = (__double2hiint(b) >> 20) & 0x7ff;
  constexpr int LOW = 1023 - TINY_EXP;
  if (xa < LOW || xb < LOW || xa == 2047 || xb == 2047 || jac::bits(g) == 0) {
    if (min(xa, xb) < LOW && max(xa, xb) < 2047 && jac::bits(a) != 0 && jac::bits(b) != 0) {
      if constexpr (TINY)
        tiny_pair<WARPS>(a, b, g, cp, cq, m, V ? V + int64_t(p) * ne : nullptr, V ? V + int64_t(q) * ne : nullptr, ne,
                         tol, rotated, red);
      else if (threadIdx.x == 0)
        rotated[TINY_AT] = 1;
    }
    return;
  }
  const int ea = (xa - 1023) & ~1, eb = (xb - 1023) & ~1;
  const float fa = jac::to_float(jac::scale_exp(a, ea)), fb = jac::to_float(jac::scale_exp(b, eb));
  const float fg = fabsf(jac::to_float(jac::scale_exp(g, (ea + eb) / 2)));
  if (!(fg > tol * sqrtf(fa * fb))) return;  // uniform over the CTA: all warps hold the same sums
  double t, c, s;
  jac::angle(g, b - a, t, c, s);
  if (threadIdx.x == 0) atomicAdd(rotated, 1);
  turn<T>(cp, cq, m, c, s);
  if (V) turn<T>(V + int64_t(p) * ne, V + int64_t(q) * ne, ne, c, s);
}

// flip[0] = 1 where the strict upper triangle of the square A carries more of its squared norm than the
// strict lower one: the columns of A^T are then the better ones to orthogonalise
__global__ void __launch_bounds__(1024) jac_orient_kernel(const double* __restrict__ A, int64_t n,
                                                          int* __restrict__ flip) {
  __shared__ float red[2][32];
  __shared__ int emax;  // entries are scaled by the largest exponent; FP32 sums do for a choice
  if (threadIdx.x == 0) emax = 0;
  __syncthreads();
  int e = 0;
  for (int64_t q = threadIdx.x; q < n * n; q += blockDim.x) {
    const int x = (__double2hiint(A[q]) >> 20) & 0x7ff;
    e = x > e && x < 2047 ? x : e;
  }
  atomicMax(&emax, e);
  __syncthreads();
  float up = 0.f, lo = 0.f;
  const int sh = emax - 1023;
  for (int64_t q = threadIdx.x; q < n * n; q += blockDim.x) {
    const int64_t i = q / n, j = q - i * n;
    const float v = jac::to_float(jac::scale_exp(A[q], sh));
    if (i < j) up = fmaf(v, v, up);
    else if (i > j) lo = fmaf(v, v, lo);
  }
  for (int o = 16; o > 0; o >>= 1) {
    up += __shfl_xor_sync(0xffffffffu, up, o);
    lo += __shfl_xor_sync(0xffffffffu, lo, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = up;
    red[1][threadIdx.x >> 5] = lo;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    up = lo = 0.f;
    for (int i = 0; i < int(blockDim.x / 32); ++i) {
      up += red[0][i];
      lo += red[1][i];
    }
    flip[0] = up > lo;
  }
}

// sigma_j = |c_j| for j < n, squared times 2^600 where the squares leave the normal range
__global__ void __launch_bounds__(JT) jac_norms_kernel(const double* __restrict__ C, int64_t m,
                                                      double* __restrict__ sig) {
  __shared__ double red[JT / 32];
  const double* c = C + int64_t(blockIdx.x) * m;
  auto sum_of_squares = [&](double f) {
    double a = 0.0;
    for (int64_t i = threadIdx.x; i < m; i += JT) {
      const double x = c[i] * f;
      a = fma(x, x, a);
    }
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = a;
    __syncthreads();
    double t = 0.0;
    for (int i = 0; i < JT / 32; ++i) t += red[i];
    return t;
  };
  double t = sum_of_squares(1.0), back = 1.0;
  if (t > 0.0 && t < 0x1p-900) {
    __syncthreads();
    t = sum_of_squares(0x1p600);
    back = 0x1p-600;
  }
  if (threadIdx.x == 0) sig[blockIdx.x] = sqrt(t) * back;
}

// order[rank] = j, descending sigma (ties by index): one CTA, rank by counting, by integer keys so that order[] is
// complete also where a sigma is NaN
__global__ void jac_rank_kernel(const double* __restrict__ sig, int n, int* __restrict__ order) {
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    const long long kj = jac::sort_key(sig[j]);
    int r = 0;
    for (int i = 0; i < n; ++i) {
      const long long ki = jac::sort_key(sig[i]);
      r += (ki > kj) || (ki == kj && i < j);
    }
    order[r] = j;
  }
}

// S[r] = sigma, U[:, r] = c_j / sigma (zero column for sigma = 0), VT[r, :] = V[:, j]
__global__ void jac_out_kernel(const double* __restrict__ C, int64_t m, const double* __restrict__ V, int ne,
                               int64_t n, const double* __restrict__ sig, const int* __restrict__ order,
                               double* __restrict__ S, double* __restrict__ U, double* __restrict__ VT) {
  const int r = blockIdx.x;
  const int j = order[r];
  const double sj = sig[j];
  if (threadIdx.x == 0 && S) S[r] = sj;
  if (U) {
    const double inv = sj > 0.0 ? 1.0 / sj : 0.0;
    const double* c = C + int64_t(j) * m;
    for (int64_t i = threadIdx.x; i < m; i += blockDim.x) U[i * n + r] = c[i] * inv;
  }
  if (VT && V) {
    const double* v = V + int64_t(j) * ne;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) VT[int64_t(r) * n + i] = v[i];
  }
}

struct JacWs {
  double *C, *V, *sig;
  int *order, *counter;
};

size_t jac_layout(int64_t m, int64_t n, bool want_v, void* base, JacWs* w) {
  const int64_t ne = n + (n & 1);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    size_t o = off;
    off += align_up(bytes);
    return o;
  };
  const size_t oC = take(size_t(m) * ne * 8), oV = take(want_v ? size_t(ne) * ne * 8 : 0),
               os = take(size_t(ne) * 8), oo = take(size_t(ne) * 4), oc = take(16);
  if (w && base) {
    char* b = static_cast<char*>(base);
    w->C = reinterpret_cast<double*>(b + oC);
    w->V = want_v ? reinterpret_cast<double*>(b + oV) : nullptr;
    w->sig = reinterpret_cast<double*>(b + os);
    w->order = reinterpret_cast<int*>(b + oo);
    w->counter = reinterpret_cast<int*>(b + oc);
  }
  return off;
}

}  // namespace
}  // namespace tnx

using namespace tnx;

extern "C" {

size_t tnx_svd_workspace_bytes(int64_t m, int64_t n, int want_vt) {
  if (m <= 0 || n <= 0 || m < n) return 0;
  return jac_layout(m, n, want_vt != 0, nullptr, nullptr);
}

int tnx_svd(const double* A, int64_t m, int64_t n, double* S, double* U, double* VT, int* sweeps_out,
            void* workspace, size_t workspace_bytes, void* stream) {
  TNX_CHECK_ARG(A && S, "null pointer");
  TNX_CHECK_ARG(m > 0 && n > 0, "non-positive dimension");
  TNX_CHECK_SHAPE(m >= n, "tnx_svd needs m >= n (got %lld x %lld); pass the transpose", (long long)m, (long long)n);
  TNX_CHECK_SHAPE(n <= (int64_t(1) << 20) && m <= (int64_t(1) << 40), "matrix too large");
  const size_t need = jac_layout(m, n, VT != nullptr, nullptr, nullptr);
  if (workspace_bytes < need || !workspace) {
    set_error("tnx_svd: workspace %zu bytes < required %zu", workspace_bytes, need);
    return TNX_ERR_WORKSPACE;
  }
  cudaStream_t st = as_stream(stream);
  JacWs w;
  jac_layout(m, n, VT != nullptr, workspace, &w);
  const int ne = int(n + (n & 1));
  int* flip = m == n && !U && !VT ? w.counter + 1 : nullptr;
  if (flip) {
    jac_orient_kernel<<<1, 1024, 0, st>>>(A, n, flip);
    TNX_LAUNCH_CHECK();
  }
  jac_init_kernel<<<152 * 4, 256, 0, st>>>(A, m, n, ne, w.C, w.V, flip);
  TNX_LAUNCH_CHECK();
  const float tol = float(sqrt(double(m)) * 2.220446049250313e-16);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3(unsigned(ne / 2));
  cfg.blockDim = dim3(m > 1024 ? 256 : 128);
  cfg.stream = st;
  cfg.attrs = at;
  int sweeps = 0, host_count = 1;
  if (ne >= 2) {
    auto kernel = m > 1024 ? jac_round_kernel<8, false> : jac_round_kernel<4, false>;
    bool tiny = false;
    TNX_CUDA(cudaMemsetAsync(w.counter + TINY_AT, 0, sizeof(int), st));
    for (; sweeps < kMaxSweeps && host_count > 0; ++sweeps) {
      TNX_CUDA(cudaMemsetAsync(w.counter, 0, sizeof(int), st));
      for (int r = 0; r < ne - 1; ++r) {
        // the first round follows a memset or another kernel: plain stream order
        cfg.numAttrs = r > 0 ? 1 : 0;
        TNX_CUDA(cudaLaunchKernelEx(&cfg, kernel, w.C, m, w.V, ne, r, tol, w.counter));
        TNX_LAUNCH_CHECK();
      }
      int seen[TINY_AT + 1];
      TNX_CUDA(cudaMemcpyAsync(seen, w.counter, sizeof(seen), cudaMemcpyDeviceToHost, st));
      TNX_CUDA(cudaStreamSynchronize(st));
      host_count = seen[0];
      if (!tiny && seen[TINY_AT]) {  // a sweep without rotations has left these pairs out
        tiny = true;
        kernel = m > 1024 ? jac_round_kernel<8, true> : jac_round_kernel<4, true>;
        host_count = 1;
      }
    }
  }
  jac_norms_kernel<<<int(n), JT, 0, st>>>(w.C, m, w.sig);
  TNX_LAUNCH_CHECK();
  jac_rank_kernel<<<1, 1024, 0, st>>>(w.sig, int(n), w.order);
  TNX_LAUNCH_CHECK();
  jac_out_kernel<<<int(n), 256, 0, st>>>(w.C, m, w.V, ne, n, w.sig, w.order, S, U, VT);
  TNX_LAUNCH_CHECK();
  if (sweeps_out) *sweeps_out = sweeps;
  if (host_count > 0) {
    TNX_CUDA(cudaStreamSynchronize(st));
    set_error("tnx_svd: %d rotations still above tolerance after %d sweeps", host_count, sweeps);
    return TNX_ERR_NOT_CONVERGED;
  }
  return TNX_OK;
}

}  // extern "C"
