// Householder QR of matrices that fit one SM's shared memory, one CTA each (FP64): the gauge moves
// of many lockstep chains (tnx_batched_gauge_move) and of small single sites.
//
// Reference: the split of MatrixProductState.split_tensor (tnpy/matrix_product_state.py:187-225).
// M (m x n, m >= n) = Q R with LAPACK's reflectors (dgeqr2): H_j = I - tau_j v v^T, v_j = 1 at the
// pivot, beta = -sign(alpha) |x|.
//
// What bounds it: 2 m n^2 - 2 n^3 / 3 FMAs for R and as many for Q at 2 FMAs per clock and SM, 215 us
// for 128 x 64, and the serial chain of a column (dot, update, norm, scalars: ~45 FP64 instructions
// of 64 clocks in one warp). So
//   * look-ahead: while the other warps apply H_j to columns j + 2 .., warp 0 applies it to column
//     j + 1 alone, takes its norm and scalars and scales v_{j+1}: one barrier a column, and the
//     chain costs nothing as long as the update is longer; the update stays off warp 0's
//     sub-partition, whose FP64 pipe would otherwise queue the chain behind it;
//   * the scalars come from an FP32 reciprocal root taken to FP64 by third-order steps, not from
//     FP64 square roots and divisions;
//   * eight lanes share a column of an update and four columns a warp: three shuffle additions per
//     four columns instead of five per column;
//   * the columns of Q are independent of each other (q_c = H_0 .. H_c e_c): four to a warp, no barrier;
//     while the batch leaves SMs idle, a cluster of up to eight CTAs repeats the factorisation (its
//     serial chain does not split) and shares the columns of Q.
// 64 chains of 128 x 64: 843 us with one warp per column, a barrier before and after the scalars and
// Q formed one reflector at a time by all warps; 372 us so, 256 chains 869 us.
#include <cooperative_groups.h>
#include <cuda_runtime.h>


#include "householder.cuh"
#include "tnx_internal.cuh"

namespace cg = cooperative_groups;

namespace tnx {
namespace {

constexpr int QS_T = 512;
constexpr int QS_W = QS_T / 32;
constexpr int QS_N = 128;  // most columns
constexpr int QS_R = 4;    // rows a lane of the pivot warp holds in registers
constexpr size_t QS_SMEM = 225 * 1024;

// column stride: 8 modulo 16 doubles, so that the two columns of a half-warp fall on distinct banks,
// where that fits
inline int qs_ld(int64_t m, int64_t n) {
  const int64_t ld = (m + 7) / 16 * 16 + 8;
  return int(size_t(2) * ld * n * sizeof(double) <= QS_SMEM ? ld : m);
}

__device__ __forceinline__ double lanes_sum(double v, int top) {
  for (int o = top; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Power of two that keeps the squares of a column in range: 1 unless alpha^2 + sigma, formed from the
// entries as they are, comes out below 2^-823 (or zero) or above 2^877. The column is then multiplied by it
// before the reflector's own factor: the product of the two overflows where the norm is subnormal
__device__ __forceinline__ double column_factor(double alpha, double sigma) {
  const int ex = (__double2hiint(fma(alpha, alpha, sigma)) >> 20) & 0x7ff;
  return ex < 200 ? 0x1p700 : (ex > 1900 ? 0x1p-600 : 1.0);
}

// trans = 0: M is the row-major m x n matrix at A_b; trans = 1: M is the transpose of the row-major
// n x m matrix at A_b. Q (m x n) goes to Q_b in the same layout (trans = 1: Q^T; Q may be A), R
// (n x n, upper triangular, row-major) to R_b.
__global__ void __launch_bounds__(QS_T) qr_small_kernel(const double* A, int64_t sA, double* Q, int64_t sQ,
                                                       double* __restrict__ Rout, int64_t sR, int m, int n, int trans,
                                                       int ld, int team) {
  extern __shared__ double qs_sm[];
  double* a = qs_sm;            // the matrix, then R above and the reflectors below the diagonal: a[j ld + i]
  double* q = qs_sm + n * ld;   // Q
  __shared__ double tau[QS_N];
  const int b = blockIdx.x / team, rank = blockIdx.x % team;
  const double* Ab = A + b * sA;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int e = tid; e < m * n; e += QS_T) {
    const int j = trans ? e / m : e % n, i = trans ? e % m : e / n;
    a[j * ld + i] = Ab[e];
    q[j * ld + i] = (i == j) ? 1.0 : 0.0;
  }
  if (team > 1) cg::this_cluster().sync();  // Q may be A: all CTAs have read it before one writes
  else __syncthreads();
  // reflector of column c, whose entries below the pivot are final; one warp
  auto reflect = [&](int c) {
    double* x = a + c * ld;
    double sg = 0.0;
    for (int i = c + 1 + lane; i < m; i += 32) sg = fma(x[i], x[i], sg);
    sg = lanes_sum(sg, 16);
    double beta, t, scale;
    const double f = column_factor(x[c], sg);
    if (f != 1.0) {
      sg = 0.0;
      for (int i = c + 1 + lane; i < m; i += 32) sg = fma(x[i] * f, x[i] * f, sg);
      sg = lanes_sum(sg, 16);
    }
    reflector(x[c] * f, sg, beta, t, scale);
    if (f == 1.0) {
      for (int i = c + 1 + lane; i < m; i += 32) x[i] *= scale;
    } else {
      beta *= f > 1.0 ? 0x1p-700 : 0x1p600;
      for (int i = c + 1 + lane; i < m; i += 32) x[i] = x[i] * f * scale;
    }
    __syncwarp();
    if (lane == 0) {
      x[c] = beta;
      tau[c] = t;
    }
  };
  if (warp == 0) reflect(0);
  __syncthreads();
  const int g = lane >> 3, h = lane & 7;
  const int worker = warp - 1 - (warp >> 2);  // of the warps outside warp 0's sub-partition (warp mod 4 != 0)
  for (int j = 0; j + 1 < n; ++j) {
    const double* v = a + j * ld;
    const double tj = tau[j];
    const bool apply = jac::bits(tj) != 0;
    if (warp == 0) {
      double* x = a + (j + 1) * ld;
      if (m - j - 1 <= 32 * QS_R) {  // the column's rows j + 1 .. in registers
        double xr[QS_R];
        const int i0 = j + 1 + lane;
#pragma unroll
        for (int r = 0; r < QS_R; ++r) xr[r] = i0 + 32 * r < m ? x[i0 + 32 * r] : 0.0;
        if (apply) {
          double vr[QS_R], w = 0.0;
#pragma unroll
          for (int r = 0; r < QS_R; ++r) vr[r] = i0 + 32 * r < m ? v[i0 + 32 * r] : 0.0;
          const double top = x[j];
#pragma unroll
          for (int r = 0; r < QS_R; ++r)
            if (j + 1 + 32 * r < m) w = fma(vr[r], xr[r], w);
          w = tj * (lanes_sum(w, 16) + top);
#pragma unroll
          for (int r = 0; r < QS_R; ++r)
            if (j + 1 + 32 * r < m) xr[r] = fma(-w, vr[r], xr[r]);
          if (lane == 0) x[j] = top - w;
        }
        const double alpha = __shfl_sync(0xffffffffu, xr[0], 0);
        double sg = lane == 0 ? 0.0 : xr[0] * xr[0], beta, t, scale;
#pragma unroll
        for (int r = 1; r < QS_R; ++r)
          if (j + 1 + 32 * r < m) sg = fma(xr[r], xr[r], sg);
        sg = lanes_sum(sg, 16);
        const double f = column_factor(alpha, sg);
        if (f == 1.0) {
          reflector(alpha, sg, beta, t, scale);
        } else {
          sg = 0.0;
#pragma unroll
          for (int r = 0; r < QS_R; ++r)
            if (r > 0 || lane > 0) sg = fma(xr[r] * f, xr[r] * f, sg);
          reflector(alpha * f, lanes_sum(sg, 16), beta, t, scale);
          beta *= f > 1.0 ? 0x1p-700 : 0x1p600;
#pragma unroll
          for (int r = 0; r < QS_R; ++r) xr[r] *= f;  // the pivot's entry becomes beta below
        }
#pragma unroll
        for (int r = 0; r < QS_R; ++r)
          if (i0 + 32 * r < m) x[i0 + 32 * r] = (r == 0 && lane == 0) ? beta : xr[r] * scale;
        if (lane == 0) tau[j + 1] = t;
      } else {
        if (apply) {
          double w = 0.0;
          for (int i = j + 1 + lane; i < m; i += 32) w = fma(v[i], x[i], w);
          const double top = x[j];  // read by every lane before lane 0 rewrites it
          w = tj * (lanes_sum(w, 16) + top);
          for (int i = j + 1 + lane; i < m; i += 32) x[i] = fma(-w, v[i], x[i]);
          if (lane == 0) x[j] = top - w;
          __syncwarp();
        }
        reflect(j + 1);
      }
    } else if (apply && (warp & 3) != 0) {
      for (int c0 = j + 2 + 4 * worker; c0 < n; c0 += 4 * (QS_W - QS_W / 4)) {
        const int c = c0 + g;
        const bool live = c < n;
        double* x = a + (live ? c : j) * ld;
        double w = 0.0;
#pragma unroll 4
        for (int i = j + 1 + h; i < m; i += 8) w = fma(v[i], x[i], w);
        const double top = x[j];
        w = tj * (lanes_sum(w, 4) + top);
        __syncwarp();
        if (live) {
#pragma unroll 4
          for (int i = j + 1 + h; i < m; i += 8) x[i] = fma(-w, v[i], x[i]);
          if (h == 0) x[j] = top - w;
        }
      }
    }
    __syncthreads();
  }
  // columns of Q, four to a warp: q_c = H_0 .. H_c e_c. Long and short ones alternate over the warps
  // of the team.
  const int items = (n + 3) / 4, workers = QS_W * team, me = warp * team + rank;
  for (int pass = 0; pass * workers < items; ++pass) {
    const int it = (pass & 1) ? (pass + 1) * workers - 1 - me : pass * workers + me;
    if (it >= items) continue;
    const int c = 4 * it + g;
    double* x = q + (c < n ? c : n - 1) * ld;
    for (int j = min(4 * it + 3, n - 1); j >= 0; --j) {
      const double* v = a + j * ld;
      const double tj = tau[j];
      const bool live = c < n && j <= c;
      double w = 0.0;
#pragma unroll 4
      for (int i = j + 1 + h; i < m; i += 8) w = fma(v[i], x[i], w);
      const double top = x[j];
      const double dot = lanes_sum(w, 4) + top;  // all lanes take part
      w = live ? tj * dot : 0.0;
      __syncwarp();
      if (live) {
#pragma unroll 4
        for (int i = j + 1 + h; i < m; i += 8) x[i] = fma(-w, v[i], x[i]);
        if (h == 0) x[j] = top - w;
      }
      __syncwarp();  // row j + 1 of the next reflector belongs to another lane
    }
  }
  __syncthreads();
  double* Qb = Q + b * sQ;
  for (int e = tid; e < m * n; e += QS_T) {
    const int j = trans ? e / m : e % n, i = trans ? e % m : e / n;
    const int p = j / 4 / workers, w = j / 4 % workers;  // whose column it is
    if (((p & 1) ? workers - 1 - w : w) % team == rank) Qb[e] = q[j * ld + i];
  }
  if (rank != 0) return;
  double* Rb = Rout + b * sR;
  for (int e = tid; e < n * n; e += QS_T) {
    const int i = e / n, c = e - i * n;
    Rb[e] = i <= c ? a[c * ld + i] : 0.0;
  }
}

}  // namespace

int qr_small(const double* A, int64_t sA, double* Q, int64_t sQ, double* R, int64_t sR, int64_t m, int64_t n, int trans,
             int batch, cudaStream_t st) {
  const int ld = qs_ld(m, n);
  static DeviceSet allowed;
  TNX_CUDA(allow_smem(qr_small_kernel, QS_SMEM, allowed));
  int team = 8;
  while (team > 1 && (batch * team > 152 || team > (n + 3) / 4)) team /= 2;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = unsigned(team);
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(unsigned(batch) * unsigned(team));
  cfg.blockDim = dim3(QS_T);
  cfg.dynamicSmemBytes = size_t(2) * ld * n * sizeof(double);
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = team > 1 ? 1 : 0;
  TNX_CUDA(cudaLaunchKernelEx(&cfg, qr_small_kernel, A, sA, Q, sQ, R, sR, int(m), int(n), trans, ld, team));
  TNX_LAUNCH_CHECK();
  return TNX_OK;
}

}  // namespace tnx
