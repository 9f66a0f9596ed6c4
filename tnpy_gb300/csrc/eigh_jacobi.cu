// Dense symmetric eigensolver, one CTA per matrix: parallel cyclic Jacobi (round-robin
// ordering, n/2 disjoint rotations per round), FP64.
//
// Used for the dense effective-Hamiltonian path of FiniteDMRG.one_site_solver
// (tnpy/finite_dmrg.py:108-110, linalg.eigh at tnpy/linalg.py:42-61, N < 200) and tSDRG blocks
// (np.linalg.eigh at tnpy/tsdrg.py:584). Jacobi is chosen for these small problems because it needs
// no tridiagonal stage, reaches full FP64 accuracy and keeps every rotation of a round
// independent, so all threads of the CTA work on one round at a time.
//
// What bounds it: an FP64 instruction holds its sub-partition's pipe for 64 clocks (2 FMAs per clock
// and SM), also in the one warp that computes a round's angles, where square roots and divisions
// are dozens of them. So
//   * A and V live in shared memory up to n = 112 (odd row stride), in the workspace above;
//   * an angle is an FP32 tangent (approximate reciprocal and root, exponents aligned by integer
//     arithmetic) taken to FP64 accuracy by two corrections against a_pq t^2 + d t - a_pq = 0, and
//     c = 1 / sqrt(1 + t^2) from an FP32 seed by one third-order step: 17 FP64 instructions, where
//     the divisions and roots took over 60;
//   * only the upper triangle of A is held and updated, a 2 x 2 block (pair k, pair l) by one thread
//     (columns, then rows, as the two-pass form), diagonal blocks by a_pp -= t a_pq, a_qq += t a_pq;
//   * the blocks that change are queued first (n <= 64), so that their threads fill whole warps: a
//     warp's FP64 instruction costs the same with one active lane, and a conserved quantity leaves
//     most blocks zero;
//   * V of round r is updated while warp 0 computes the angles of round r + 1, by the warps of the
//     other three sub-partitions, so it does not wait for warp 0's pipe: two barriers a round.
// 128 tSDRG blocks of 64 x 64 (one conserved quantity): 3.02 ms with A and V in the workspace, exact
// angles and full passes over A, 1.00 ms so (1.25 ms without the queue); 64 random dense 64 x 64
// matrices 7.9 and 3.0 ms; one 199 x 199 156 and 128 ms.
#include <cuda_runtime.h>

#include <algorithm>

#include "jacobi.cuh"
#include "tnx_internal.cuh"

namespace tnx {
namespace {

constexpr int EJ_THREADS = 512;
constexpr int EJ_MAX_SWEEPS = 40;
constexpr int EJ_MAX_N = 1024;   // largest matrix
constexpr int EJ_SHARED_N = 112;  // largest matrix whose A and V fit in shared memory

// row stride in shared memory: odd, so that a column's entries fall on distinct banks
__host__ __device__ constexpr int ej_ld(int n) { return n | 1; }
constexpr size_t ej_smem_bytes(int n) { return size_t(2) * n * ej_ld(n) * sizeof(double); }

// A: matrix b at A + offsets[b], leading dimension lds[b] (or sizes[b] when lds == null).
// work (matrices beyond EJ_SHARED_N): per matrix 2*max_size^2 doubles (copy of A and the rotation
// accumulator V).
__global__ void __launch_bounds__(EJ_THREADS) jacobi_eigh_kernel(
    const double* __restrict__ A_all, const int64_t* __restrict__ offsets, const int* __restrict__ sizes,
    const int* __restrict__ lds, int n_uniform, int ld_uniform, int max_size, int keep,
    double* __restrict__ evals, double* __restrict__ evecs, double* __restrict__ work) {
  extern __shared__ double ej_sm[];
  const int b = blockIdx.x;
  const int n = sizes ? sizes[b] : n_uniform;
  const int lda = lds ? lds[b] : (sizes ? n : ld_uniform);
  const double* Ain = A_all + (offsets ? offsets[b] : int64_t(b) * ld_uniform * n_uniform);
  const bool shared = max_size <= EJ_SHARED_N;
  const int ld = shared ? ej_ld(n) : n;
  double* A = shared ? ej_sm : work + size_t(b) * 2 * size_t(max_size) * max_size;
  double* V = A + (shared ? size_t(n) * ld : size_t(max_size) * max_size);
  const int tid = threadIdx.x, nt = EJ_THREADS, lane = tid & 31, warp = tid >> 5;
  constexpr int NW = EJ_THREADS / 32;

  // rotations of the current and the previous round
  __shared__ double sc[2][EJ_MAX_N / 2], ss[2][EJ_MAX_N / 2];
  __shared__ int16_t sp[2][EJ_MAX_N / 2], sq[2][EJ_MAX_N / 2];
  __shared__ double red[NW];
  __shared__ uint16_t queue[32 * 31 / 2];  // blocks to update (n <= 64)
  __shared__ int s_count;
  __shared__ int s_any[2];  // whether the round rotates anything
  __shared__ int s_rot;     // whether the sweep did
  __shared__ double s_fro;

  if (n <= 0) return;
  double fro = 0.0;
  for (int e = tid; e < n * n; e += nt) {
    const int i = e / n, j = e - i * n;
    const double v = Ain[size_t(i) * lda + j];
    A[i * ld + j] = v;  // the strict lower triangle is not used
    V[i * ld + j] = (i == j) ? 1.0 : 0.0;
    fro = fma(v, v, fro);
  }
  for (int o = 16; o > 0; o >>= 1) fro += __shfl_xor_sync(0xffffffffu, fro, o);
  if (lane == 0) red[warp] = fro;
  __syncthreads();
  if (tid == 0) {
    double t = 0.0;
    for (int w = 0; w < NW; ++w) t += red[w];
    s_fro = sqrt(t);
  }
  __syncthreads();
  // off-diagonal entries below the rounding noise of the rotations (~eps*||A||) are left alone,
  // so that a sweep can end without any rotation (compared as integers: both are positive)
  const long long floor_bits = __double_as_longlong(1e-300 + 2e-16 * s_fro);

  const int np = n + (n & 1), npairs = np / 2;
  // V <- V J with the rotations of buffer u, pairs slot, slot + slots, ...
  auto update_v = [&](int u, int slot, int slots) {
    for (int l = slot; l < npairs; l += slots) {
      const double s = ss[u][l];
      if (jac::bits(s) == 0) continue;
      const double c = sc[u][l];
      const int p = sp[u][l], q = sq[u][l];
      for (int j = lane; j < n; j += 32) {
        const double vp = V[j * ld + p], vq = V[j * ld + q];
        V[j * ld + p] = fma(c, vp, -s * vq);
        V[j * ld + q] = fma(s, vp, c * vq);
      }
    }
  };
  auto at = [&](int i, int j) -> double& { return i < j ? A[i * ld + j] : A[j * ld + i]; };
  // whether block (k, l) changes: one of the pairs rotates and the block is not all zero (a conserved
  // quantity keeps most of A exactly zero)
  auto active = [&](int u, int k, int l) {
    if ((jac::bits(ss[u][k]) | jac::bits(ss[u][l])) == 0) return false;
    const int pk = sp[u][k], qk = sq[u][k], pl = sp[u][l], ql = sq[u][l];
    const bool row2 = qk < n, col2 = ql < n;  // the padding player of an odd n has no entries
    unsigned long long z = jac::bits(at(pk, pl));
    if (col2) z |= jac::bits(at(pk, ql));
    if (row2) z |= jac::bits(at(qk, pl));
    if (row2 && col2) z |= jac::bits(at(qk, ql));
    return z != 0;
  };
  auto update_block = [&](int u, int k, int l) {
    const double sk = ss[u][k], sl = ss[u][l];
    const int pk = sp[u][k], qk = sq[u][k], pl = sp[u][l], ql = sq[u][l];
    const bool row2 = qk < n, col2 = ql < n;
    double a = at(pk, pl), b2 = col2 ? at(pk, ql) : 0.0, c2 = row2 ? at(qk, pl) : 0.0,
           d2 = row2 && col2 ? at(qk, ql) : 0.0;
    if (jac::bits(sl)) {
      const double c = sc[u][l], a0 = a, c0 = c2;
      a = fma(c, a0, -sl * b2);
      b2 = fma(sl, a0, c * b2);
      c2 = fma(c, c0, -sl * d2);
      d2 = fma(sl, c0, c * d2);
    }
    if (jac::bits(sk)) {
      const double c = sc[u][k], a0 = a, b0 = b2;
      a = fma(c, a0, -sk * c2);
      c2 = fma(sk, a0, c * c2);
      b2 = fma(c, b0, -sk * d2);
      d2 = fma(sk, b0, c * d2);
    }
    at(pk, pl) = a;
    if (col2) at(pk, ql) = b2;
    if (row2) at(qk, pl) = c2;
    if (row2 && col2) at(qk, ql) = d2;
  };
  if (n > 1) {
    bool pending = false;  // the previous round's rotations still to be applied to V
    int u = 0;
    for (int sweep = 0; sweep < EJ_MAX_SWEEPS; ++sweep) {
      if (tid == 0) s_rot = 0;
      if (npairs > 32) __syncthreads();  // other warps than the first set it too
      for (int r = 0; r < np - 1; ++r, u ^= 1) {
        // rotations of this round by the first warps, V of the round before by the others: with few
        // pairs warp 0 alone, and V on the other three sub-partitions (warp mod 4 != 0)
        if (tid < ((npairs + 31) & ~31)) {
          const int k = tid;
          bool rot = false;
          if (k < npairs) {
            int p, q;
            jac::pair_of(k, r, np, p, q);
            double c = 1.0, s = 0.0;
            if (q < n) {
              const double apq = A[p * ld + q];
              const long long ab = __double_as_longlong(apq) & 0x7fffffffffffffffLL;
              if (ab > floor_bits && ab < 0x7ff0000000000000LL) {
                double t;
                const double app = A[p * ld + p], aqq = A[q * ld + q];
                jac::angle(apq, aqq - app, t, c, s);
                A[p * ld + p] = fma(-t, apq, app);
                A[q * ld + q] = fma(t, apq, aqq);
                A[p * ld + q] = 0.0;
                rot = true;
              }
            }
            sp[u][k] = int16_t(p);
            sq[u][k] = int16_t(q);
            sc[u][k] = c;
            ss[u][k] = s;
          }
          const bool any = __any_sync(0xffffffffu, rot);
          if (npairs <= 32) {
            if (tid == 0) {
              s_any[u] = any;
              s_count = 0;
            }
          }
          if (any && lane == 0) s_rot = 1;
        }
        if (npairs <= 32) {
          if (pending && (warp & 3) != 0) update_v(u ^ 1, warp - 1 - (warp >> 2), NW - NW / 4);
        } else if (pending) {
          update_v(u ^ 1, warp, NW);
        }
        __syncthreads();
        if (npairs <= 32 && !s_any[u]) {  // nothing rotates: no update of A, nor of V
          pending = false;
          continue;
        }
        pending = true;
        // A <- J^T A J above the diagonal: blocks (rows of pair k, columns of pair l), k < l; rows k
        // and npairs - 1 - k together have npairs - 1 blocks
        for (int w = warp; w < (npairs + 1) / 2; w += NW) {
          const int k2 = npairs - 1 - w, n1 = npairs - 1 - w, n2 = k2 > w ? w : 0;
          for (int x = lane; x < ((n1 + n2 + 31) & ~31); x += 32) {
            const int k = x < n1 ? w : k2, l = x < n1 ? w + 1 + x : k2 + 1 + (x - n1);
            const bool act = x < n1 + n2 && active(u, k, l);
            if (npairs > 32) {
              if (act) update_block(u, k, l);
              continue;
            }
            const unsigned m = __ballot_sync(0xffffffffu, act);
            int base = 0;
            if (lane == 0 && m) base = atomicAdd(&s_count, __popc(m));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (act) queue[base + __popc(m & ((1u << lane) - 1))] = uint16_t(k << 8 | l);
          }
        }
        if (npairs <= 32) {
          __syncthreads();
          for (int i = tid; i < s_count; i += nt) update_block(u, queue[i] >> 8, queue[i] & 255);
        }
        __syncthreads();
      }
      const int rot = s_rot;
      __syncthreads();  // every thread has read the flag before the next sweep clears it
      if (rot == 0) break;
    }
    if (pending) update_v(u ^ 1, warp, NW);
    __syncthreads();
  }
  // ascending order: rank of each diagonal entry (ties broken by index), by its sortable bits
  __shared__ int16_t rank[EJ_MAX_N];
  auto key = [&](int i) { return jac::sort_key(A[i * ld + i]); };
  double* ev_out = evals + size_t(b) * keep;
  double* vec_out = evecs + size_t(b) * max_size * keep;
  for (int i = tid; i < n; i += nt) {
    const long long di = key(i);
    int rk = 0;
    for (int j = 0; j < n; ++j) {
      const long long dj = key(j);
      rk += (dj < di) || (dj == di && j < i);
    }
    rank[i] = int16_t(rk);
    if (rk < keep) ev_out[rk] = A[i * ld + i];
  }
  __syncthreads();
  for (int e = tid; e < n * n; e += nt) {
    const int row = e / n, i = e - row * n;
    if (rank[i] < keep) vec_out[size_t(row) * keep + rank[i]] = V[row * ld + i];
  }
}

}  // namespace

namespace {
int launch_jacobi(const double* A, const int64_t* offsets, const int* sizes, const int* lds, int n, int ld, int batch,
                  int max_size, int keep, double* evals, double* evecs, double* work, cudaStream_t st) {
  const size_t smem = max_size <= EJ_SHARED_N ? ej_smem_bytes(max_size) : 0;
  static DeviceSet allowed;
  TNX_CUDA(allow_smem(jacobi_eigh_kernel, ej_smem_bytes(EJ_SHARED_N), allowed));
  jacobi_eigh_kernel<<<batch, EJ_THREADS, smem, st>>>(A, offsets, sizes, lds, n, ld, max_size, keep, evals, evecs,
                                                      work);
  TNX_LAUNCH_CHECK();
  return TNX_OK;
}
}  // namespace

int eigh_small_f64_ld(const double* A, const int64_t* offsets, const int* sizes, const int* lds,
                      int batch, int max_size, int keep, double* evals, double* evecs, double* work,
                      cudaStream_t st) {
  if (batch <= 0) return TNX_OK;
  return launch_jacobi(A, offsets, sizes, lds, 0, 0, batch, max_size, keep, evals, evecs, work, st);
}

int eigh_small_f64_uniform(const double* A, int n, int ld, int keep, double* evals, double* evecs,
                           double* work, cudaStream_t st) {
  return launch_jacobi(A, nullptr, nullptr, nullptr, n, ld, 1, n, keep, evals, evecs, work, st);
}

int eigh_small_f64(double* A, const int64_t* offsets, const int* sizes, int batch, int max_size,
                   int keep, double* evals, double* evecs, double* work, cudaStream_t st) {
  return eigh_small_f64_ld(A, offsets, sizes, nullptr, batch, max_size, keep, evals, evecs, work, st);
}

}  // namespace tnx

using namespace tnx;

extern "C" {

size_t tnx_eigh_batched_workspace_bytes(int batch, int max_size, int keep) {
  (void)keep;
  if (batch <= 0 || max_size <= 0) return 0;
  return align_up(size_t(batch) * 2 * size_t(max_size) * max_size * sizeof(double));
}

int tnx_eigh_batched(double* A, const int64_t* offsets, const int* sizes, int batch, int max_size,
                     int keep, double* evals, double* evecs, void* workspace, size_t workspace_bytes,
                     void* stream) {
  TNX_CHECK_ARG(A && offsets && sizes && evals && evecs, "null pointer");
  TNX_CHECK_ARG(batch >= 0 && max_size > 0 && keep > 0 && keep <= max_size,
                "bad batch/max_size/keep (%d, %d, %d)", batch, max_size, keep);
  TNX_CHECK_SHAPE(max_size <= 1024, "eigh: matrices larger than 1024 are not supported (got %d)",
                  max_size);
  size_t need = align_up(size_t(batch) * 2 * size_t(max_size) * max_size * sizeof(double));
  if (workspace_bytes < need || !workspace) {
    set_error("tnx_eigh_batched: workspace %zu bytes < required %zu", workspace_bytes, need);
    return TNX_ERR_WORKSPACE;
  }
  if (batch == 1 && keep == 1 && max_size <= 64)  // one small matrix, lowest pair
    return rr_lowest_f64(A, max_size, max_size, evals, evecs, as_stream(stream));
  return eigh_small_f64(A, offsets, sizes, batch, max_size, keep, evals, evecs,
                        static_cast<double*>(workspace), as_stream(stream));
}

}  // extern "C"

// ---------------------------------------------------------------------------------------
// Lowest eigenpair of small symmetric matrices (n <= 64), one CTA each (256 threads, 1024 above 32 rows): the
// Davidson Rayleigh-Ritz problem and the dense effective Hamiltonians of the chain ends.
//
// An FP64 instruction holds its sub-partition's pipe for 64 clocks on GB300 (2 FMAs per clock and
// SM), an FP32 one for one, so the Jacobi sweeps run in FP32 and the lowest pair is then refined
// against the FP64 matrix,
//   s <- s - sum_{j != 0} v_j (v_j . r) / (lambda_j - theta),  r = A s - theta s,
// which contracts the error by ~(FP32 eigenvector error) / (relative gap) per step; three steps reach
// FP64 accuracy where the lowest eigenvalue is well apart, a closer one takes up to seven, while the
// corrections shrink (gaps of 1e-3 of the norm, 24 rows: residual 7e-14 after three, 2e-16 so).
// theta = s^T A s is FP64.
// Only s, r, theta and the norm are FP64: the correction's relative error of ~1e-6 is what the
// FP32 eigenvectors leave it anyway, and the next step works it off.
//
// A round of the sweep is two barriers long: the angles (one thread per pair), then every 2 x 2
// block (pair k, pair l) of A <- J^T A J by one thread, columns first as in the two-pass form, so
// each entry sees the operations of the two-pass form; a round without a rotation ends at the first
// barrier. A random 24 x 24 matrix: 211 us with a pass and a barrier each for columns, rows and zeroing,
// exact divisions and the correction in FP64, 80 us so; 64 x 64: 1.90 ms and
// 0.39 ms (0.47 ms by 256 threads).
// ---------------------------------------------------------------------------------------
namespace tnx {
namespace {

constexpr int RW_MAX = 64;

constexpr int RR_G = 8;      // warps that share a product of the refinement
constexpr int RR_STEPS = 7;  // most corrections

// x 2^-e; zero for zero and where it would be subnormal
__device__ __forceinline__ double rr_scale(double x, int e) {
  return (__double2hiint(x) & 0x7ff00000) == 0 ? 0.0 : jac::scale_exp(x, e);
}

// FP32 rounding keeps regenerating off-diagonal entries at ~6e-8 |A|_F, so the sweeps
// stop once every off-diagonal entry is below 1e-6 |A|_F; the FP64 steps take it from there.
// Block b solves the matrix at A + b sA into eval[b sE], evec + b sV, and returns at
// once when active is given and active[b] == 0. With `sizes` (count > 0), block b solves the leading block
// of sizes.n[b] rows of A instead of n, and where[b] is the index at which the sweeps left the lowest value.
// The matrix is taken times the power of two that brings its largest entry below one (exact): sweeps and corrections are
// FP32's. One with Inf or NaN has NaN for its pair.
template <int RR_T>
__global__ void __launch_bounds__(RR_T) rr_lowest_kernel(const double* __restrict__ A, int n, int ld,
                                                         double* __restrict__ eval, double* __restrict__ evec,
                                                         int64_t sA, int64_t sE, int64_t sV,
                                                         const int* __restrict__ active, const RrSizes sizes,
                                                         double* __restrict__ where) {
  if (active && !active[blockIdx.x]) return;
  if (sizes.count > 0) n = sizes.n[blockIdx.x];
  A += int64_t(blockIdx.x) * sA;
  eval += int64_t(blockIdx.x) * sE;
  evec += int64_t(blockIdx.x) * sV;
  extern __shared__ double sm_d[];
  const int nf = n + 1;
  double* Ad = sm_d;                                      // n x (n+1) FP64
  double* s = Ad + n * nf;                                // n
  double* rp = s + n;                                     // partial products, RR_G x n
  float* Af = reinterpret_cast<float*>(rp + RR_G * n);       // n x (n+1) FP32
  float* Vf = Af + n * nf;                                // n x (n+1) FP32
  float* rf = Vf + n * nf;                                // n: residual
  float* fp = rf + n;                                     // partial projections, RR_G x n
  __shared__ float4 rot[32];  // c, s and (as integers) p, q of a pair
  __shared__ float red[RR_T / 32];
  __shared__ double redd[RR_T / 32];
  __shared__ unsigned s_max[RR_T / 32];
  __shared__ int s_imin;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned mx = 0;
  for (int e = tid; e < n * n; e += RR_T) {
    const int i = e / n, j = e - i * n;
    const double v = A[int64_t(i) * ld + j];
    Ad[i * nf + j] = v;
    Vf[i * nf + j] = (i == j) ? 1.f : 0.f;
    mx = max(mx, unsigned(__double2hiint(v)) & 0x7fffffffu);
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  if (lane == 0) s_max[warp] = mx;
  __syncthreads();
  for (int w = 0; w < RR_T / 32; ++w) mx = max(mx, s_max[w]);
  if (mx >= 0x7ff00000u) {
    if (tid == 0) eval[0] = __longlong_as_double(0x7ff8000000000000LL);
    if (tid < n) evec[tid] = __longlong_as_double(0x7ff8000000000000LL);
    if (where && tid == 0) where[blockIdx.x] = 0.0;
    return;
  }
  const int ex = int(mx >> 20) - 1022;
  float fro = 0.f;
  for (int e = tid; e < n * n; e += RR_T) {
    const int i = e / n, j = e - i * n;
    const double v = rr_scale(Ad[i * nf + j], ex);
    const float f = float(v);
    Ad[i * nf + j] = v;
    Af[i * nf + j] = f;
    fro += f * f;
  }
  for (int o = 16; o > 0; o >>= 1) fro += __shfl_xor_sync(0xffffffffu, fro, o);
  if (lane == 0) red[warp] = fro;
  __syncthreads();
  fro = 0.f;
  for (int w = 0; w < RR_T / 32; ++w) fro += red[w];
  fro = sqrtf(fro);
  const float thresh = 1e-6f * fro;
  if (n > 1) {
    const int np = n + (n & 1), npairs = np / 2;
    const int tx = tid & 15, ty = tid >> 4;
    for (int sweep = 0; sweep < 30; ++sweep) {
      bool any = false;
      for (int rnd = 0; rnd < np - 1; ++rnd) {
        bool turns = false;
        if (tid < npairs) {
          int p, q;
          jac::pair_of(tid, rnd, np, p, q);
          float c = 1.f, sn = 0.f;
          if (q < n) {
            const float apq = Af[p * nf + q], app = Af[p * nf + p], aqq = Af[q * nf + q];
            if (fabsf(apq) > thresh) {  // |th| < 1e6 then, and th^2 is far from overflow
              // approximate reciprocals (a few ulp): the FP64 steps correct what the sweeps leave
              const float th = __fdividef(0.5f * (aqq - app), apq);
              const float h2 = fmaf(th, th, 1.f);
              const float t = copysignf(__fdividef(1.f, fmaf(h2, rsqrtf(h2), fabsf(th))), th);
              c = rsqrtf(fmaf(t, t, 1.f));
              sn = t * c;
              turns = true;
            }
          }
          rot[tid] = make_float4(c, sn, __int_as_float(p), __int_as_float(q));
        }
        if (!__syncthreads_or(turns)) continue;  // nothing to apply: straight to the next round's angles
        any = true;
        // A <- J^T (A J): block (rows of pair k, columns of pair l); the padding player of an odd n
        // (index n) has no entries
        for (int k = ty; k < npairs; k += RR_T / 16) {
          const float4 rk = rot[k];
          const float sk = rk.y, ck = rk.x;
          const int pk = __float_as_int(rk.z), qk = __float_as_int(rk.w);
          for (int l = tx; l < npairs; l += 16) {
            const float4 rl = rot[l];
            const float sl = rl.y, cl = rl.x;
            if (sk == 0.f && sl == 0.f) continue;
            const int pl = __float_as_int(rl.z), ql = __float_as_int(rl.w);
            const bool row2 = qk < n, col2 = ql < n;
            float* r0 = Af + pk * nf;
            float* r1 = Af + qk * nf;
            float a = r0[pl], b = col2 ? r0[ql] : 0.f, c = row2 ? r1[pl] : 0.f, d = row2 && col2 ? r1[ql] : 0.f;
            if (sl != 0.f) {
              const float a1 = cl * a - sl * b, b1 = sl * a + cl * b;
              const float c1 = cl * c - sl * d, d1 = sl * c + cl * d;
              a = a1; b = b1; c = c1; d = d1;
            }
            if (sk != 0.f) {
              const float a1 = ck * a - sk * c, c1 = sk * a + ck * c;
              const float b1 = ck * b - sk * d, d1 = sk * b + ck * d;
              a = a1; b = b1; c = c1; d = d1;
            }
            if (k == l) b = c = 0.f;  // the entry this rotation removes
            r0[pl] = a;
            if (col2) r0[ql] = b;
            if (row2) r1[pl] = c;
            if (row2 && col2) r1[ql] = d;
          }
        }
        // V <- V J
        for (int l = ty; l < npairs; l += RR_T / 16) {
          const float4 rl = rot[l];
          const float sl = rl.y, cl = rl.x;
          if (sl == 0.f) continue;
          const int pl = __float_as_int(rl.z), ql = __float_as_int(rl.w);
          for (int j = tx; j < n; j += 16) {
            const float va = Vf[j * nf + pl], vb = Vf[j * nf + ql];
            Vf[j * nf + pl] = cl * va - sl * vb;
            Vf[j * nf + ql] = sl * va + cl * vb;
          }
        }
        __syncthreads();
      }
      if (!any) break;
    }
  }
  // lowest FP32 eigenvalue (the first of equal ones), by warp 0
  if (warp == 0) {
    int im = lane < n ? lane : 0;
    float dm = Af[im * nf + im];
    if (lane + 32 < n && Af[(lane + 32) * nf + lane + 32] < dm) {
      im = lane + 32;
      dm = Af[im * nf + im];
    }
    for (int o = 16; o > 0; o >>= 1) {
      const float od = __shfl_xor_sync(0xffffffffu, dm, o);
      const int oi = __shfl_xor_sync(0xffffffffu, im, o);
      if (od < dm || (od == dm && oi < im)) {
        dm = od;
        im = oi;
      }
    }
    if (lane == 0) s_imin = im;
  }
  __syncthreads();
  const int imin = s_imin;
  if (where && tid == 0) where[blockIdx.x] = double(imin);
  for (int i = tid; i < n; i += RR_T) s[i] = double(Vf[i * nf + imin]);
  __syncthreads();
  const float floor = 1e-6f * fro;
  // warp g takes columns g, g + RR_G, ... of a product; the partial sums are added in group order
  auto sum_d = [&](int i) {
    double t = rp[i];
#pragma unroll
    for (int g = 1; g < RR_G; ++g) t += rp[g * n + i];
    return t;
  };
  auto sum_f = [&](int i) {
    float t = fp[i];
#pragma unroll
    for (int g = 1; g < RR_G; ++g) t += fp[g * n + i];
    return t;
  };
  int last = 3;         // the step that ends it
  float dd_prev = 0.f;  // squared norm of the correction before
  for (int step = 0;; ++step) {
    // y = A s, then |s|^2 and s . y together (n <= 64: the entries sit in warps 0 and 1)
    for (int i = warp < RR_G ? lane : n; i < n; i += 32) {
      double acc = 0.0;
      for (int j = warp; j < n; j += RR_G) acc = fma(Ad[i * nf + j], s[j], acc);
      rp[warp * n + i] = acc;
    }
    __syncthreads();
    double yi = 0.0, si = 0.0;
    if (warp < 2) {
      if (tid < n) {
        yi = sum_d(tid);
        si = s[tid];
      }
      double nn = 0.0, sy = 0.0;
      if (warp * 32 < n) {
        nn = si * si;
        sy = si * yi;
        for (int o = 16; o > 0; o >>= 1) {
          nn += __shfl_xor_sync(0xffffffffu, nn, o);
          sy += __shfl_xor_sync(0xffffffffu, sy, o);
        }
      }
      if (lane == 0) {
        redd[warp] = nn;
        redd[2 + warp] = sy;
      }
    }
    __syncthreads();
    const double nn = redd[0] + redd[1];
    const double inv = jac::rsqrt_exact(nn);  // nn is 1 to FP32 accuracy
    const double theta = (redd[2] + redd[3]) * (inv * inv);
    if (tid < n) s[tid] = si * inv;
    if (step == last) {
      if (tid == 0) eval[0] = scale_pow2(theta, ex);
      break;
    }
    if (tid < n) rf[tid] = float(fma(-theta, si, yi) * inv);
    __syncthreads();
    // f_j = (v_j . r) / (l_j - theta); (near-)degenerate partners keep f_j = 0
    for (int j = warp < RR_G ? lane : n; j < n; j += 32) {
      float acc = 0.f;
      for (int i = warp; i < n; i += RR_G) acc = fmaf(Vf[i * nf + j], rf[i], acc);
      fp[warp * n + j] = acc;
    }
    __syncthreads();
    for (int j = tid; j < n; j += RR_T) {
      const float den = float(double(Af[j * nf + j]) - theta);
      const float dot = sum_f(j);
      rf[j] = (j != imin && fabsf(den) > floor) ? dot / den : 0.f;  // the floor of a zero matrix is zero
    }
    __syncthreads();
    if (step > 0) {  // every warp the same sum
      float dd = lane < n ? rf[lane] * rf[lane] : 0.f;
      if (lane + 32 < n) dd = fmaf(rf[lane + 32], rf[lane + 32], dd);
      for (int o = 16; o > 0; o >>= 1) dd += __shfl_xor_sync(0xffffffffu, dd, o);
      // the next correction would be about dd / dd_prev of this one: another step while that is above rounding
      if (step == last - 1 && last < RR_STEPS && dd < 0.25f * dd_prev && dd * (dd / dd_prev) > 1e-32f) ++last;
      dd_prev = dd;
    }
    for (int i = warp < RR_G ? lane : n; i < n; i += 32) {
      float acc = 0.f;
      for (int j = warp; j < n; j += RR_G) acc = fmaf(Vf[i * nf + j], rf[j], acc);
      fp[warp * n + i] = acc;
    }
    __syncthreads();
    for (int i = tid; i < n; i += RR_T) s[i] -= double(sum_f(i));
    __syncthreads();
  }
  if (tid < n) evec[tid] = s[tid];  // the thread's own entry
}

}  // namespace

size_t rr_lowest_smem(int n) {
  return size_t(n) * (n + 1) * 16 + size_t(n) * ((1 + RR_G) * 8 + (1 + RR_G) * 4);
}

namespace {
int launch_rr(const double* A, int n, int ld, int64_t sA, double* eval, int64_t sE, double* evec, int64_t sV, int batch,
              const int* active, const RrSizes& sizes, double* where, cudaStream_t st) {
  if (n > RW_MAX) {
    set_error("rr_lowest_f64: n=%d > %d", n, RW_MAX);
    return TNX_ERR_SHAPE;
  }
  if (batch <= 0) return TNX_OK;
  static DeviceSet allowed;
  TNX_CUDA(allow_smem(rr_lowest_kernel<1024>, rr_lowest_smem(RW_MAX), allowed));
  profile_mark(KF_EIGH, st, true);
  // the blocks of a round, (n / 2)^2 of them and n^2 / 4 entries of V twice, by a thread each
  if (n <= 32)
    rr_lowest_kernel<256><<<batch, 256, rr_lowest_smem(n), st>>>(A, n, ld, eval, evec, sA, sE, sV, active, sizes, where);
  else
    rr_lowest_kernel<1024><<<batch, 1024, rr_lowest_smem(n), st>>>(A, n, ld, eval, evec, sA, sE, sV, active, sizes, where);
  profile_mark(KF_EIGH, st, false);
  TNX_LAUNCH_CHECK();
  return TNX_OK;
}
}  // namespace

int rr_lowest_f64(const double* A, int n, int ld, double* eval, double* evec, cudaStream_t st) {
  return launch_rr(A, n, ld, 0, eval, 0, evec, 0, 1, nullptr, RrSizes{}, nullptr, st);
}

int rr_lowest_f64_batched(const double* A, int n, int ld, int64_t sA, double* eval, int64_t sE, double* evec,
                          int64_t sV, int batch, const int* active, cudaStream_t st) {
  return launch_rr(A, n, ld, sA, eval, sE, evec, sV, batch, active, RrSizes{}, nullptr, st);
}

int rr_lowest_f64_leading(const double* A, int ld, const RrSizes& sizes, double* eval, double* evec, int64_t sV,
                          double* where, cudaStream_t st) {
  return launch_rr(A, *std::max_element(sizes.n, sizes.n + sizes.count), ld, 0, eval, 1, evec, sV, sizes.count, nullptr,
                   sizes, where, st);
}

}  // namespace tnx

// ---------------------------------------------------------------------------------------
// The lowest pair by way of a tridiagonal form (n <= 64), for a Davidson's Rayleigh-Ritz steps: four
// warps. Only one pair is wanted, so FP32 finds that one: Householder reflectors (a lane holds a row in
// registers, one warp per 32 rows; as many warps apply the reflectors to the rows of Q at the same
// time), 32 Sturm sequences at a time around the lowest eigenvalue, and its vector from the twisted
// factorisation of T - lambda. FP64 then refines the pair against the given matrix,
//   s <- s - Q x,  (T - lambda) x = Q^T r without row and column k,  r = A s - theta s,
// where k is the twist index: T - lambda without it is positive definite, and its factors are there
// already. A step contracts the error by ~(FP32 error) / gap, and the steps go on until the next one
// would be below FP64 rounding (two as a rule, six at most). Only s, r, theta and the norm are FP64;
// the correction's relative error of ~1e-6 is what T and Q leave it anyway. theta gains s . r, whose
// FP32 rounding shrinks with r. A random 24 x 24 matrix: 80 us in the kernel above, 27 us here; 64 x 64:
// 385 and 76 us; the mean over a chi = 32 eigensolve's 68 problems 45 and 20 us.
//
// The vector's largest entry is positive. The sweeps above give their vector the same sign, and leave its
// value at that entry's index, where the square of the entry is at least 0.99 (none of 4.7 million random problems of
// 3 to 24 rows differed; 1 in 13000 did between 0.9 and 0.99).
// ---------------------------------------------------------------------------------------
namespace tnx {
namespace {

constexpr int RT_T = 128;

__device__ __forceinline__ float rr_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int NR>
__global__ void __launch_bounds__(RT_T) rr_tri_kernel(const double* __restrict__ A, int n, int ld,
                                                      double* __restrict__ eval, double* __restrict__ evec) {
  constexpr int LR = NR / 32;  // rows per lane of one warp
  constexpr int QS = NR + 1;   // row stride of Q (conflict-free along rows and columns)
  extern __shared__ double sm_d[];
  const int nf = n + 1;
  double* Ad = sm_d;                                   // n x (n+1) FP64
  float* Vs = reinterpret_cast<float*>(Ad + n * nf);   // reflector k in row k
  float* Q = Vs + NR * NR;                             // first the scaled matrix, then Q
  __shared__ __align__(16) float xrow[2][NR], pw[NR];
  __shared__ float td[NR], te[NR], cs[NR], red[2];
  __shared__ float2 tde[NR];                           // diagonal, square of the off-diagonal before it
  __shared__ float2 fm[2][NR];                         // pivots' reciprocals and multipliers, from both ends
  __shared__ float piv[2][NR], gv[NR], yv[NR], zv[NR], dv[NR];
  __shared__ double sd[NR], rp[3][NR];
  __shared__ unsigned s_max[RT_T / 32];
  __shared__ int s_done;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  // the matrix, and the power of two that brings its Frobenius norm to at most one
  unsigned mx = 0;
  for (int i = warp; i < n; i += RT_T / 32)
    for (int j = lane; j < n; j += 32) {
      const double v = A[int64_t(i) * ld + j];
      Ad[i * nf + j] = v;
      mx = max(mx, unsigned(__double2hiint(v)) & 0x7fffffffu);
    }
  mx = __reduce_max_sync(0xffffffffu, mx);
  if (lane == 0) s_max[warp] = mx;
  __syncthreads();
  mx = max(max(s_max[0], s_max[1]), max(s_max[2], s_max[3]));
  if (mx >= 0x7ff00000u) {  // Inf or NaN, which the scaling below would make finite
    if (tid == 0) eval[0] = __longlong_as_double(0x7ff8000000000000LL);
    if (tid < n) evec[tid] = __longlong_as_double(0x7ff8000000000000LL);
    return;
  }
  const int ex = int(mx >> 20) - 1022 + (NR == 32 ? 5 : 6);
  for (int i = warp; i < NR; i += RT_T / 32)
#pragma unroll
    for (int j = lane; j < NR; j += 32)
      Q[i * QS + j] = i < n && j < n ? jac::to_float(rr_scale(Ad[i * nf + j], ex)) : 0.f;
  __syncthreads();

  // ---- tridiagonal form: warps [0, LR) hold the rows of A, warps [LR, 2 LR) those of Q
  const bool is_a = warp < LR, is_q = !is_a && warp < 2 * LR;
  const int row = (is_a ? warp : warp - LR) * 32 + lane;
  float a[NR];
  if (is_a) {
#pragma unroll
    for (int j = 0; j < NR; ++j) a[j] = Q[row * QS + j];
  } else {
#pragma unroll
    for (int j = 0; j < NR; ++j) a[j] = j == row ? 1.f : 0.f;
  }
  auto sync_a = [] {  // among the warps of A
    if (LR == 1) __syncwarp();
    else __syncthreads();
  };
  for (int k = 0; k < n; ++k) {
    float* xr = xrow[k & 1];
    if (is_a && row == k) {
#pragma unroll
      for (int j = 0; j < NR; j += 4) *reinterpret_cast<float4*>(xr + j) = make_float4(a[j], a[j + 1], a[j + 2], a[j + 3]);
    }
    sync_a();
    if (tid == 0) td[k] = xr[k];
    if (k >= n - 2) {
      if (tid == 0) te[k] = k == n - 2 ? xr[n - 1] : 0.f;
      continue;
    }
    float vi = 0.f, c = 0.f;
    if (is_a) {  // the reflector, by each warp of A for itself
      const float alpha = xr[k + 1];
      float sq = 0.f;
#pragma unroll
      for (int j = lane; j < NR; j += 32) sq += j > k + 1 ? xr[j] * xr[j] : 0.f;
      sq = rr_sum(sq);
      float beta = alpha;
      if (sq > 1e-22f) {  // entries below 1e-11 of the norm count as zero
        const float h = fmaf(alpha, alpha, sq), nr = h * rsqrtf(h);
        beta = -copysignf(nr, alpha);
        c = __fdividef(1.f, nr * (nr + fabsf(alpha)));
        vi = row > k + 1 ? xr[row] : (row == k + 1 ? alpha - beta : 0.f);
      }
      Vs[k * NR + row] = vi;
      if (tid == 0) {
        te[k] = beta;
        cs[k] = c;
      }
    }
    __syncthreads();
    const float* v = Vs + k * NR;
    auto times_v = [&] {
      float p0 = 0.f, p1 = 0.f, p2 = 0.f, p3 = 0.f;
#pragma unroll
      for (int j = 0; j < NR; j += 4) {
        const float4 x = *reinterpret_cast<const float4*>(v + j);
        p0 = fmaf(a[j], x.x, p0);
        p1 = fmaf(a[j + 1], x.y, p1);
        p2 = fmaf(a[j + 2], x.z, p2);
        p3 = fmaf(a[j + 3], x.w, p3);
      }
      return (p0 + p1) + (p2 + p3);
    };
    float p = 0.f, dot = 0.f;
    if (is_a) {
      p = c * times_v();
      dot = rr_sum(p * vi);
    }
    if (LR == 2) {
      if (is_a) pw[row] = p;
      if (is_a && lane == 0) red[warp] = dot;
      __syncthreads();
    }
    if (is_a) {
      if (LR == 1) {
        const float wi = fmaf(-0.5f * c * dot, vi, p);
        pw[row] = wi;
        __syncwarp();
#pragma unroll
        for (int j = 0; j < NR; j += 4) {
          const float4 x = *reinterpret_cast<const float4*>(v + j), w = *reinterpret_cast<const float4*>(pw + j);
          a[j] = fmaf(-vi, w.x, fmaf(-wi, x.x, a[j]));
          a[j + 1] = fmaf(-vi, w.y, fmaf(-wi, x.y, a[j + 1]));
          a[j + 2] = fmaf(-vi, w.z, fmaf(-wi, x.z, a[j + 2]));
          a[j + 3] = fmaf(-vi, w.w, fmaf(-wi, x.w, a[j + 3]));
        }
      } else {
        const float kk = 0.5f * c * (red[0] + red[1]), wi = fmaf(-kk, vi, p);
        const float ui = fmaf(-kk, vi, wi);  // a - v_i w_j - w_i v_j = a - v_i p_j - (w_i - K v_i) v_j
#pragma unroll
        for (int j = 0; j < NR; j += 4) {
          const float4 x = *reinterpret_cast<const float4*>(v + j), q = *reinterpret_cast<const float4*>(pw + j);
          a[j] = fmaf(-vi, q.x, fmaf(-ui, x.x, a[j]));
          a[j + 1] = fmaf(-vi, q.y, fmaf(-ui, x.y, a[j + 1]));
          a[j + 2] = fmaf(-vi, q.z, fmaf(-ui, x.z, a[j + 2]));
          a[j + 3] = fmaf(-vi, q.w, fmaf(-ui, x.w, a[j + 3]));
        }
      }
    } else if (is_q) {  // Q <- Q (1 - c v v^T)
      const float y = cs[k] * times_v();
#pragma unroll
      for (int j = 0; j < NR; j += 4) {
        const float4 x = *reinterpret_cast<const float4*>(v + j);
        a[j] = fmaf(-y, x.x, a[j]);
        a[j + 1] = fmaf(-y, x.y, a[j + 1]);
        a[j + 2] = fmaf(-y, x.z, a[j + 2]);
        a[j + 3] = fmaf(-y, x.w, a[j + 3]);
      }
    }
  }
  if (is_q) {  // the scaled matrix in its place was read before the loop's first barrier
#pragma unroll
    for (int j = 0; j < NR; ++j) Q[row * QS + j] = a[j];
  }
  __syncthreads();

  // ---- lowest eigenvalue of T and the factors, by warp 0
  double sv[LR], theta = 0.0;
  float z[LR], nrm = 0.f;
  int kt = 0;
  auto q_times = [&](const float* x, int i) {  // row i of Q
    float t0 = 0.f, t1 = 0.f, t2 = 0.f, t3 = 0.f;
#pragma unroll
    for (int j = 0; j < NR; j += 4) {
      t0 = fmaf(Q[i * QS + j], x[j], t0);
      t1 = fmaf(Q[i * QS + j + 1], x[j + 1], t1);
      t2 = fmaf(Q[i * QS + j + 2], x[j + 2], t2);
      t3 = fmaf(Q[i * QS + j + 3], x[j + 3], t3);
    }
    return (t0 + t1) + (t2 + t3);
  };
  if (warp == 0) {
    float lo = 3e38f, hi = 3e38f;
#pragma unroll
    for (int i = lane; i < NR; i += 32) {
      if (i < n) {
        const float dd = td[i], e0 = i > 0 ? te[i - 1] : 0.f, off = fabsf(e0) + fabsf(te[i]);
        lo = fminf(lo, dd - off);
        hi = fminf(hi, dd);
        nrm = fmaxf(nrm, fabsf(dd) + off);
        tde[i] = make_float2(dd, e0 * e0);
      }
      zv[i] = dv[i] = gv[i] = 0.f;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fminf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      nrm = fmaxf(nrm, __shfl_xor_sync(0xffffffffu, nrm, o));
    }
    __syncwarp();
    lo -= 1e-6f * nrm;
    // 33^5 parts of at most twice the norm: 5e-8 of it. A sequence of leading minors (rescaled every
    // four, the norm is at most one) stays positive below the lowest eigenvalue.
    for (int pass = 0; pass < 5; ++pass) {
      const float h = (hi - lo) * (1.f / 33.f), x = fmaf(h, float(lane + 1), lo);
      float p0 = 1.f, p1 = 1.f, mn = 1.f;
      for (int i = 0; i < n; i += 4) {
        const float f = __uint_as_float((254u << 23) - (__float_as_uint(p1) & 0x7f800000u));
        p0 *= f;
        p1 *= f;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (i + u < n) {
            const float2 t = tde[i + u];
            const float p2 = fmaf(t.x - x, p1, -t.y * p0);
            p0 = p1;
            p1 = p2;
            mn = fminf(mn, p2);
          }
        }
      }
      const unsigned below = __ballot_sync(0xffffffffu, mn > 0.f);
      const int f = below == 0xffffffffu ? 32 : __ffs(~below) - 1;  // first lane at or above it
      const float l0 = lo;
      if (f > 0) lo = fmaf(h, float(f), l0);
      if (f < 32) hi = fmaf(h, float(f + 1), l0);
    }
    // pivots of T - lo from the top (lane 0) and from the bottom (lane 1); those before the twist are
    // positive, and below the rounding of T they mean nothing
    const float floor = fmaxf(1e-6f * nrm, 1e-30f);
    if (lane < 2) {
      float prev = 0.f;  // off-diagonal squared / pivot
      for (int t = 0; t < n; ++t) {
        const int i = lane == 0 ? t : n - 1 - t;
        const float p = (td[i] - lo) - prev;
        const float r = __fdividef(1.f, fmaxf(p, floor));
        const float e = lane == 0 ? te[i] : (i > 0 ? te[i - 1] : 0.f);
        piv[lane][i] = p;
        fm[lane][i] = make_float2(r, -e * r);
        prev = e * e * r;
      }
    }
    __syncwarp();
    float gm = 3e38f;
#pragma unroll
    for (int i = lane; i < NR; i += 32)
      if (i < n) {
        const float g = fabsf(piv[0][i] + piv[1][i] - (td[i] - lo));
        if (g < gm) {
          gm = g;
          kt = i;
        }
      }
    for (int o = 16; o > 0; o >>= 1) {
      const float og = __shfl_xor_sync(0xffffffffu, gm, o);
      const int oi = __shfl_xor_sync(0xffffffffu, kt, o);
      if (og < gm || (og == gm && oi < kt)) {
        gm = og;
        kt = oi;
      }
    }
    if (lane < 2) {
      float x = 1.f;
      if (lane == 0) zv[kt] = 1.f;
      const int m = lane == 0 ? kt : n - 1 - kt, step = lane == 0 ? -1 : 1;
#pragma unroll 4
      for (int t = 1; t <= m; ++t) {
        const int i = kt + t * step;
        x *= fm[lane][i].y;
        zv[i] = x;
      }
    }
    __syncwarp();
    float zz = 0.f;
#pragma unroll
    for (int u = 0; u < LR; ++u) {
      z[u] = zv[lane + 32 * u];
      zz = fmaf(z[u], z[u], zz);
    }
    const float zi = rsqrtf(rr_sum(zz));
    __syncwarp();
#pragma unroll
    for (int u = 0; u < LR; ++u) zv[lane + 32 * u] = z[u] *= zi;
    __syncwarp();
    float sf[LR], big = -1.f, val = 0.f;
#pragma unroll
    for (int u = 0; u < LR; ++u) {
      sf[u] = q_times(zv, lane + 32 * u);
      if (fabsf(sf[u]) > big) {
        big = fabsf(sf[u]);
        val = sf[u];
      }
    }
    int at = lane;
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, big, o), ov = __shfl_xor_sync(0xffffffffu, val, o);
      const int oa = __shfl_xor_sync(0xffffffffu, at, o);
      if (ob > big || (ob == big && oa < at)) {
        big = ob;
        val = ov;
        at = oa;
      }
    }
#pragma unroll
    for (int u = 0; u < LR; ++u) sd[lane + 32 * u] = sv[u] = jac::to_double(copysignf(1.f, val) * sf[u]);
    theta = rr_scale(jac::to_double(lo), -ex);
  }
  __syncthreads();

  // ---- refinement: warps 1-3 form A s, warp 0 the norm and the correction
  float dn_prev = 1.f;
  for (int step = 0; step < 6; ++step) {
    double nn = 0.0;
    if (warp > 0) {
#pragma unroll
      for (int i = lane; i < NR; i += 32)
        if (i < n) {
          double acc = 0.0;
          for (int j = warp - 1; j < n; j += 3) acc = fma(Ad[i * nf + j], sd[j], acc);
          rp[warp - 1][i] = acc;
        }
    } else {
#pragma unroll
      for (int u = 0; u < LR; ++u) nn = fma(sv[u], sv[u], nn);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) nn += __shfl_xor_sync(0xffffffffu, nn, o);
    }
    __syncthreads();
    if (warp == 0) {
      const float inn = __fdividef(1.f, jac::to_float(nn));
      float rf[LR], sf[LR], rho = 0.f;
#pragma unroll
      for (int u = 0; u < LR; ++u) {
        const int i = lane + 32 * u;
        const double y = i < n ? (rp[0][i] + rp[1][i]) + rp[2][i] : 0.0;
        rf[u] = jac::to_float(rr_scale(fma(-theta, sv[u], y), ex));
        sf[u] = jac::to_float(sv[u]);
        rho = fmaf(rf[u], sf[u], rho);
      }
      rho = rr_sum(rho) * inn;
      theta += rr_scale(jac::to_double(rho), -ex);
#pragma unroll
      for (int u = 0; u < LR; ++u) yv[lane + 32 * u] = fmaf(-rho, sf[u], rf[u]);
      __syncwarp();
#pragma unroll
      for (int u = 0; u < LR; ++u) {  // Q^T r
        float t0 = 0.f, t1 = 0.f;
#pragma unroll
        for (int i = 0; i < NR; i += 2) {
          t0 = fmaf(Q[i * QS + lane + 32 * u], yv[i], t0);
          t1 = fmaf(Q[(i + 1) * QS + lane + 32 * u], yv[i + 1], t1);
        }
        gv[lane + 32 * u] = t0 + t1;
      }
      __syncwarp();
      if (lane < 2) {  // lane 0 the rows above the twist, lane 1 those below
        const int m = lane == 0 ? kt : n - 1 - kt, first = lane == 0 ? 0 : n - 1, up = lane == 0 ? 1 : -1;
        float x = 0.f, mu = 0.f;
#pragma unroll 4
        for (int t = 0; t < m; ++t) {
          const int i = first + t * up;
          x = fmaf(mu, x, gv[i]);
          const float2 f = fm[lane][i];
          yv[i] = x * f.x;
          mu = f.y;
        }
        x = 0.f;
#pragma unroll 4
        for (int t = 1; t <= m; ++t) {
          const int i = kt - t * up;
          x = fmaf(fm[lane][i].y, x, yv[i]);
          dv[i] = x;
        }
        if (lane == 0) dv[kt] = 0.f;
      }
      __syncwarp();
      float d[LR], zd = 0.f, dd = 0.f;
#pragma unroll
      for (int u = 0; u < LR; ++u) {
        d[u] = dv[lane + 32 * u];
        zd = fmaf(d[u], z[u], zd);
      }
      zd = rr_sum(zd);
      __syncwarp();
#pragma unroll
      for (int u = 0; u < LR; ++u) {
        d[u] = fmaf(-zd, z[u], d[u]);
        dd = fmaf(d[u], d[u], dd);
        dv[lane + 32 * u] = d[u];
      }
      dd = rr_sum(dd);
      __syncwarp();
      const double inv = jac::rsqrt_exact(nn);
      const bool last = step == 5;
#pragma unroll
      for (int u = 0; u < LR; ++u) {
        const double c = last ? 0.0 : jac::to_double(q_times(dv, lane + 32 * u));
        sd[lane + 32 * u] = sv[u] = (sv[u] - c) * inv;
      }
      // the next correction would be about dd / dn_prev; rho's own rounding is 1e-7 of it
      const float dn = sqrtf(dd);
      const bool done = last || (fabsf(rho) <= 1e-9f * nrm && (dd <= 2e-16f * dn_prev || dn <= 1e-15f));
      dn_prev = dn;
      if (lane == 0) s_done = done;
      if (done) {
        if (lane == 0) eval[0] = theta;
#pragma unroll
        for (int u = 0; u < LR; ++u)
          if (lane + 32 * u < n) evec[lane + 32 * u] = sv[u];
      }
    }
    __syncthreads();
    if (s_done) break;
  }
}

size_t rr_tri_smem(int n, int nr) { return size_t(n) * (n + 1) * 8 + size_t(nr) * (2 * nr + 1) * 4; }

}  // namespace

int rr_lowest_tri(const double* A, int n, int ld, double* eval, double* evec, cudaStream_t st) {
  if (n > RW_MAX) {
    set_error("rr_lowest_tri: n=%d > %d", n, RW_MAX);
    return TNX_ERR_SHAPE;
  }
  profile_mark(KF_EIGH, st, true);
  if (n <= 32) {
    rr_tri_kernel<32><<<1, RT_T, rr_tri_smem(n, 32), st>>>(A, n, ld, eval, evec);
  } else {
    static DeviceSet allowed;
    TNX_CUDA(allow_smem(rr_tri_kernel<64>, rr_tri_smem(RW_MAX, 64), allowed));
    rr_tri_kernel<64><<<1, RT_T, rr_tri_smem(n, 64), st>>>(A, n, ld, eval, evec);
  }
  profile_mark(KF_EIGH, st, false);
  TNX_LAUNCH_CHECK();
  return TNX_OK;
}

}  // namespace tnx
