// FP64 contraction kernels of the one-site effective Hamiltonian and the environment
// updates (the plain FP64 form), plus the C ABI entry points that sequence them.
//
// Reference: Environment.one_site_matvec (tnpy/matrix_product_state.py:411-440),
// update_left / update_right (:296-336), one_site_full_matrix (:372-409).
//
// Every contraction is L x MPS -> MPO -> R split into two GEMMs (K = chi and K = chi*D)
// around a small dense MPO step (K = D*d), i.e. 4*chi^3*D*d + 2*chi^2*D^2*d^2 flops.
#include <cooperative_groups.h>

#include <algorithm>
#include <cuda_runtime.h>

#include <cstring>
#include <mutex>

#include "tnx_internal.cuh"
#include "wcontract.cuh"

namespace cg = cooperative_groups;

namespace tnx {

// ---------------------------------------------------------------------------------
// FP64 SIMT GEMM. GB300 issues 2 FP64 FMAs per clock and SM (one warp instruction occupies its
// sub-partition's pipe for 64 clocks), so the pipe is the bound at every shape, a tile of any
// size keeps it fed, and the time of a product is the FMA count of the busiest SM: what matters
// is that the work spreads over all 152 SMs with little padding. Hence three tiles (64 x 64,
// 32 x 32, 16 x 16) and a split of K over the CTAs of a thread-block cluster, whose partial tiles
// are summed through distributed shared memory in rank order (deterministic, no workspace);
// f64_plan picks the pair with the least FMAs on the busiest SM. The next 16-deep K slab is
// loaded into registers while the current one is multiplied. Threads own interleaved outputs, so
// the shared-memory reads of a warp hit distinct banks.
// ---------------------------------------------------------------------------------
namespace {
constexpr int GB_K = 16;

template <bool TA, bool TB, int BM, int BN, int NT>
__global__ void __launch_bounds__(NT) gemm_f64_kernel(int64_t M, int64_t N, int64_t K, double alpha,
                                                     const double* __restrict__ A, int64_t lda,
                                                     int64_t sa, const double* __restrict__ B,
                                                     int64_t ldb, int64_t sb, double beta,
                                                     double* __restrict__ C, int64_t ldc,
                                                     int64_t sc, int64_t k_total,
                                                     const int* __restrict__ bmask, int nsplit, int64_t kslice) {
  constexpr int TY = NT / 16, RI = BM / TY, RJ = BN / 16;  // outputs per thread
  constexpr int LA = BM * GB_K / NT, LB = BN * GB_K / NT;  // slab elements per thread
  static_assert(BM % TY == 0 && BN % 16 == 0 && LA * NT == BM * GB_K && LB * NT == BN * GB_K, "FP64 GEMM tile");
  constexpr int STAGE = GB_K * (BM + 1 + BN + 1), TILE = BM * BN;
  __shared__ double sm[STAGE > TILE ? STAGE : TILE];  // slab, then the partial tile of a split product
  double(*As)[BM + 1] = reinterpret_cast<double(*)[BM + 1]>(sm);
  double(*Bs)[BN + 1] = reinterpret_cast<double(*)[BN + 1]>(sm + GB_K * (BM + 1));
  const int64_t bz = blockIdx.z / nsplit;
  const int rank = int(blockIdx.z % nsplit);  // = the CTA's rank in its 1 x 1 x nsplit cluster
  if (bmask && !bmask[bz]) return;  // a batch entry the caller masked out (all of its cluster)
  A += bz * sa;
  B += bz * sb;
  C += bz * sc;
  const int64_t m0 = int64_t(blockIdx.y) * BM, n0 = int64_t(blockIdx.x) * BN;
  // split-K mode (k_total > 0): batch index bz owns K range [bz*K, min((bz+1)*K, k_total))
  if (k_total > 0) {
    const int64_t rem = k_total - bz * K;
    K = rem < K ? rem : K;
  }
  const int64_t kb = rank * kslice, ke = kb + kslice < K ? kb + kslice : K;
  const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
  double acc[RI][RJ];
#pragma unroll
  for (int i = 0; i < RI; ++i)
#pragma unroll
    for (int j = 0; j < RJ; ++j) acc[i][j] = 0.0;

  double pa[LA], pb[LB];
  // global -> registers for the slab at k0 (zero outside the matrix and the slice); consecutive
  // threads walk the unit-stride index
  auto fetch = [&](int64_t k0) {
#pragma unroll
    for (int r = 0; r < LA; ++r) {
      const int e = tid + r * NT;
      const int mm = TA ? e % BM : e / GB_K, kk = TA ? e / BM : e % GB_K;
      const int64_t gm = m0 + mm, gk = k0 + kk;
      pa[r] = (gm < M && gk < ke) ? (TA ? A[gk * lda + gm] : A[gm * lda + gk]) : 0.0;
    }
#pragma unroll
    for (int r = 0; r < LB; ++r) {
      const int e = tid + r * NT;
      const int nn = TB ? e / GB_K : e % BN, kk = TB ? e % GB_K : e / BN;
      const int64_t gn = n0 + nn, gk = k0 + kk;
      pb[r] = (gn < N && gk < ke) ? (TB ? B[gn * ldb + gk] : B[gk * ldb + gn]) : 0.0;
    }
  };
  auto stage = [&]() {
#pragma unroll
    for (int r = 0; r < LA; ++r) {
      const int e = tid + r * NT;
      As[TA ? e / BM : e % GB_K][TA ? e % BM : e / GB_K] = pa[r];
    }
#pragma unroll
    for (int r = 0; r < LB; ++r) {
      const int e = tid + r * NT;
      Bs[TB ? e % GB_K : e / BN][TB ? e / GB_K : e % BN] = pb[r];
    }
  };
  if (kb < ke) {
    fetch(kb);
    stage();
    __syncthreads();
    for (int64_t k0 = kb; k0 < ke; k0 += GB_K) {
      const bool more = k0 + GB_K < ke;
      if (more) fetch(k0 + GB_K);
      const int kn = ke - k0 < GB_K ? int(ke - k0) : GB_K;  // no FMAs on the padding of a short slab
#pragma unroll 4
      for (int kk = 0; kk < kn; ++kk) {
        double a[RI], b[RJ];
#pragma unroll
        for (int i = 0; i < RI; ++i) a[i] = As[kk][ty + TY * i];
#pragma unroll
        for (int j = 0; j < RJ; ++j) b[j] = Bs[kk][tx + 16 * j];
#pragma unroll
        for (int i = 0; i < RI; ++i)
#pragma unroll
          for (int j = 0; j < RJ; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
      }
      __syncthreads();
      if (more) {
        stage();
        __syncthreads();
      }
    }
  }
  auto put = [&](int64_t gm, int64_t gn, double v) {
    if (gm >= M || gn >= N) return;
    v *= alpha;
    if (beta != 0.0) v = fma(beta, C[gm * ldc + gn], v);
    C[gm * ldc + gn] = v;
  };
  if (nsplit == 1) {
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
      for (int j = 0; j < RJ; ++j) put(m0 + ty + TY * i, n0 + tx + 16 * j, acc[i][j]);
    return;
  }
  // the slices' partial tiles, summed in rank order; each rank finishes its share of the elements
  cg::cluster_group cluster = cg::this_cluster();
#pragma unroll
  for (int i = 0; i < RI; ++i)
#pragma unroll
    for (int j = 0; j < RJ; ++j) sm[(ty + TY * i) * BN + tx + 16 * j] = acc[i][j];
  cluster.sync();
  for (int e = rank * NT + tid; e < TILE; e += NT * nsplit) {
    double v = 0.0;
    for (int r = 0; r < nsplit; ++r) v += cluster.map_shared_rank(sm, r)[e];
    put(m0 + e / BN, n0 + e % BN, v);
  }
  cluster.sync();  // no CTA leaves while another may still read its tile
}

// Tile (64, 32 or 16 rows and columns) and K split of one product. The cost of a candidate is the
// number of FMA clocks of the busiest SM, ceil(CTAs / 152) * tile * slice / 2, plus its fixed part
// (launch, first loads, the cluster's sum). Measured (GB300, per call): 402 x 168 x 840, 886 us
// with 64 x 64 tiles (21 CTAs) and 120 us planned (286 of 16 x 16; the pipe alone: 90 us);
// 64 x 32 x 160, 172 us (one CTA) and 7.7 us planned; 512^3, 538 and 237 us; 2048 x 1024 x 5120,
// 20.6 ms without the prefetch and 17.4 ms with it (1.235 of 1.26 TFLOP/s).
struct F64Plan {
  int tile, nsplit;
  int64_t kslice;
  double clocks;  // estimate
};

F64Plan f64_plan(int64_t m, int64_t n, int64_t k, int64_t batch) {
  static const int tiles[3] = {64, 32, 16};
  static const int splits[4] = {1, 2, 4, 8};  // 8: the largest portable cluster
  F64Plan best{64, 1, (k + GB_K - 1) / GB_K * GB_K, 0.0};
  double best_cost = 1e300;
  for (int t : tiles) {
    const int64_t my = (m + t - 1) / t, nx = (n + t - 1) / t;
    if (my > 65535 && t < 64) continue;  // beyond the grid's y limit
    for (int s : splits) {
      if (batch * s > 65535 || (s > 1 && t == 64)) break;
      const int64_t ks = ((k + s - 1) / s + GB_K - 1) / GB_K * GB_K;
      if (s > 1 && ks * (s - 1) >= k) break;  // an empty slice
      const double ctas = double(my) * double(nx) * double(batch) * s;
      const double waves = double(int64_t((ctas + 151) / 152));
      const double per = double(t) * t * double(ks < k ? ks : k) / 2.0;
      // fixed clocks per CTA: first slab, store (and the cluster's barriers and sum)
      const double cost = waves * (per + t * t / 2.0) + 2000.0 + (s > 1 ? 3000.0 + waves * t * t / 2.0 : 0.0);
      if (cost < best_cost) {
        best_cost = cost;
        best = {t, s, ks, cost};
      }
    }
  }
  return best;
}

template <int BM, int BN, int NT>
int launch_f64(bool ta, bool tb, const F64Plan& p, dim3 grid, int64_t m, int64_t n, int64_t k, double alpha,
               const double* A, int64_t lda, int64_t sa, const double* B, int64_t ldb, int64_t sb, double beta,
               double* C, int64_t ldc, int64_t sc, cudaStream_t st, int64_t k_total, const int* bmask) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = unsigned(p.nsplit);
  cfg.gridDim = grid;
  cfg.blockDim = dim3(NT);
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = p.nsplit > 1 ? 1 : 0;
  auto go = [&](auto kernel) {
    return cudaLaunchKernelEx(&cfg, kernel, m, n, k, alpha, A, lda, sa, B, ldb, sb, beta, C, ldc, sc, k_total, bmask,
                              p.nsplit, p.kslice);
  };
  if (!ta && !tb) TNX_CUDA(go(gemm_f64_kernel<false, false, BM, BN, NT>));
  else if (ta && !tb) TNX_CUDA(go(gemm_f64_kernel<true, false, BM, BN, NT>));
  else if (!ta && tb) TNX_CUDA(go(gemm_f64_kernel<false, true, BM, BN, NT>));
  else TNX_CUDA(go(gemm_f64_kernel<true, true, BM, BN, NT>));
  return TNX_OK;
}
}  // namespace

bool f64_cheaper(int64_t m, int64_t n, int64_t k, int nsplit) {
  // a double-FP32 product of K slices of kc in 32 x 32 tiles: 560 clocks a step of K in a tile's chain, 200 of an SM's
  // time once several tiles share it; partial sums in memory where split
  const int64_t kc = (k + nsplit - 1) / nsplit;
  const double tiles = double((m + 31) / 32) * double((n + 31) / 32) * nsplit;
  const double df = std::max(560.0, tiles / 152.0 * 200.0) * double(kc) + 4000.0 + (nsplit > 1 ? 6000.0 : 0.0);
  return f64_plan(m, n, k, 1).clocks < df;
}

int gemm_f64(bool ta, bool tb, int64_t m, int64_t n, int64_t k, double alpha, const double* A,
             int64_t lda, int64_t sa, const double* B, int64_t ldb, int64_t sb, double beta,
             double* C, int64_t ldc, int64_t sc, int64_t batch, cudaStream_t st, int64_t k_total,
             const int* bmask) {
  if (m <= 0 || n <= 0 || batch <= 0) return TNX_OK;
  if (k <= 0) {
    // C = beta * C; only the beta == 0 case is used here
    TNX_CHECK_ARG(beta == 0.0, "gemm_f64: k == 0 with beta != 0 not supported");
    for (int64_t b = 0; b < batch; ++b)
      for (int64_t r = 0; r < m; ++r) TNX_CUDA(cudaMemsetAsync(C + b * sc + r * ldc, 0, n * 8, st));
    return TNX_OK;
  }
  TNX_CHECK_SHAPE(batch <= 65535, "gemm_f64: batch %lld > 65535", (long long)batch);
  const F64Plan p = f64_plan(m, n, k, batch);
  dim3 grid((unsigned)((n + p.tile - 1) / p.tile), (unsigned)((m + p.tile - 1) / p.tile),
            (unsigned)(batch * p.nsplit));
  TNX_CHECK_SHAPE(grid.y <= 65535, "gemm_f64: m too large");
  profile_mark(KF_F64_GEMM, st, true);
  if (p.tile == 64)
    TNX_TRY((launch_f64<64, 64, 256>(ta, tb, p, grid, m, n, k, alpha, A, lda, sa, B, ldb, sb, beta, C, ldc, sc, st,
                                     k_total, bmask)));
  else if (p.tile == 32)
    TNX_TRY((launch_f64<32, 32, 128>(ta, tb, p, grid, m, n, k, alpha, A, lda, sa, B, ldb, sb, beta, C, ldc, sc, st,
                                     k_total, bmask)));
  else
    TNX_TRY((launch_f64<16, 16, 128>(ta, tb, p, grid, m, n, k, alpha, A, lda, sa, B, ldb, sb, beta, C, ldc, sc, st,
                                     k_total, bmask)));
  profile_mark(KF_F64_GEMM, st, false);
  profile_work(KF_F64_GEMM, 2.0 * double(m) * n * k * batch, 8.0 * batch * (double(m) * k + double(k) * n + double(m) * n));
  TNX_LAUNCH_CHECK();
  return TNX_OK;
}

namespace {
// C = alpha * sum_z P[z] + beta * C (P: nsplit partial m x n row-major products)
__global__ void splitk_reduce_kernel(const double* __restrict__ P, int nsplit, int64_t m, int64_t n, double alpha,
                                     double beta, double* __restrict__ C, int64_t ldc) {
  const int64_t mn = m * n;
  for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < mn; e += int64_t(gridDim.x) * blockDim.x) {
    double acc = 0.0;
    for (int z = 0; z < nsplit; ++z) acc += P[z * mn + e];
    const int64_t i = e / n, j = e % n;
    double v = alpha * acc;
    if (beta != 0.0) v = fma(beta, C[i * ldc + j], v);
    C[i * ldc + j] = v;
  }
}
}  // namespace

int gemm_f64_splitk(bool ta, bool tb, int64_t m, int64_t n, int64_t k, double alpha, const double* A, int64_t lda,
                    const double* B, int64_t ldb, double beta, double* C, int64_t ldc, int nsplit, double* part,
                    cudaStream_t st, bool df, bool alone) {
  // FP64 products split K inside gemm_f64 (clusters), without partials in memory; `alone`: nothing of note runs beside
  // the product, so that clusters are scheduled at once
  if (!df || nsplit <= 1 || (alone && f64_cheaper(m, n, k, nsplit)))
    return gemm_fp64_class(df && nsplit <= 1, ta, tb, m, n, k, alpha, A, lda, 0, B, ldb, 0, beta, C, ldc, 0, 1, st);
  const int64_t kc = (k + nsplit - 1) / nsplit;
  nsplit = int((k + kc - 1) / kc);
  const int64_t sa = ta ? kc * lda : kc, sb = tb ? kc : kc * ldb;
  TNX_TRY(gemm_fp64_class(df, ta, tb, m, n, kc, 1.0, A, lda, sa, B, ldb, sb, 0.0, part, n, m * n, nsplit, st, k));
  int64_t blocks = (m * n + 255) / 256;
  if (blocks > 152 * 8) blocks = 152 * 8;
  splitk_reduce_kernel<<<unsigned(blocks < 1 ? 1 : blocks), 256, 0, st>>>(part, nsplit, m, n, alpha, beta, C, ldc);
  TNX_LAUNCH_CHECK();
  return TNX_OK;
}

// MPO step of one site (wcontract.cuh)
int wcontract_left(const double* T1, const double* W, double* T2, int64_t chi_l, int64_t d,
                   int64_t chi_r, int64_t dl, int64_t dr, cudaStream_t st) {
  TNX_CHECK_SHAPE(dl * d <= 64 && dr * d <= 64, "MPO bond too large (dl*d, dr*d <= %d)", 64);
  return wc::launch_left<double>(T1, 0, W, 0, wc::OutF64{T2}, 0, chi_l, d, chi_r, dl, dr, chi_r * dr, 1, nullptr, st);
}

int wcontract_right(const double* T1, const double* W, double* T2, int64_t chi_l, int64_t d,
                    int64_t chi_r, int64_t dl, int64_t dr, cudaStream_t st) {
  TNX_CHECK_SHAPE(dl * d <= 64 && dr * d <= 64, "MPO bond too large (dl*d, dr*d <= %d)", 64);
  return wc::launch_right<double>(T1, 0, W, 0, T2, 0, chi_l, d, chi_r, dl, dr, 1, st);
}

int64_t matvec1_scratch_elems(int64_t chi_l, int64_t d, int64_t chi_r, int64_t dl, int64_t dr) {
  int64_t a = dl * chi_l * d * chi_r, b = chi_l * d * chi_r * dr;
  return a > b ? a : b;
}

bool use_oz(int64_t m, int64_t n, int64_t k) {
  // the tensor-core FP64-class GEMM pays five launches of operand slicing: large products only
  return m >= 256 && n >= 64 && k >= 128 && double(m) * double(n) * double(k) >= double(1 << 27);
}

int gemm_fp64_class_oz(bool df, bool ta, bool tb, int64_t m, int64_t n, int64_t k, double alpha, const double* A,
                       int64_t lda, const double* B, int64_t ldb, double beta, double* C, int64_t ldc, void* oz_ws,
                       size_t oz_bytes, cudaStream_t st) {
  if (df && oz_ws && use_oz(m, n, k) && oz_bytes >= gemm_oz_workspace_bytes(m, n, k)) {
    // FP64-class engine, autotuned per shape: 0 tcgen05 Ozaki GEMM, 1 double-FP32 SIMT GEMM
    auto run = [&](int v) -> int {
      if (v == 0) return gemm_oz(ta, tb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, oz_ws, oz_bytes, st);
      return gemm_fp64_class(true, ta, tb, m, n, k, alpha, A, lda, 0, B, ldb, 0, beta, C, ldc, 0, 1, st);
    };
    const TuneKey key{2, int64_t(ta) * 2 + int64_t(tb), m, n, k, 0};
    return autotuned(key, 2, 0, beta == 0.0, st, run);
  }
  return gemm_fp64_class(df, ta, tb, m, n, k, alpha, A, lda, 0, B, ldb, 0, beta, C, ldc, 0, 1, st);
}

size_t matvec1_oz_bytes(int64_t chi_l, int64_t d, int64_t chi_r, int64_t dl, int64_t dr) {
  size_t a = use_oz(dl * chi_l, d * chi_r, chi_l) ? gemm_oz_workspace_bytes(dl * chi_l, d * chi_r, chi_l) : 0;
  size_t b = use_oz(chi_l * d, chi_r, chi_r * dr) ? gemm_oz_workspace_bytes(chi_l * d, chi_r, chi_r * dr) : 0;
  return a > b ? a : b;
}

int matvec1_f64(const double* L, const double* W, const double* R, const double* x, double* y,
                int64_t chi_l, int64_t d, int64_t chi_r, int64_t dl, int64_t dr, double* T1,
                double* T2, cudaStream_t st, bool df, void* oz_ws, size_t oz_bytes) {
  // T1[(w,a'),(s,c)] = sum_a L[a,(w,a')] x[a,(s,c)]
  TNX_TRY(gemm_fp64_class_oz(df, true, false, dl * chi_l, d * chi_r, chi_l, 1.0, L, dl * chi_l, x, d * chi_r, 0.0,
                             T1, d * chi_r, oz_ws, oz_bytes, st));
  TNX_TRY(wcontract_left(T1, W, T2, chi_l, d, chi_r, dl, dr, st));
  // y[(a',s'),c'] = sum_{(c,v)} T2[(a',s'),(c,v)] R[(c,v),c']
  TNX_TRY(gemm_fp64_class_oz(df, false, false, chi_l * d, chi_r, chi_r * dr, 1.0, T2, chi_r * dr, R, chi_r, 0.0, y,
                             chi_r, oz_ws, oz_bytes, st));
  return TNX_OK;
}

// ---------------------------------------------------------------------------------
// diag(H_eff) and dense H_eff
// ---------------------------------------------------------------------------------
namespace {
__global__ void diag1_kernel(const double* __restrict__ L, const double* __restrict__ W,
                             const double* __restrict__ R, double* __restrict__ diag, int64_t chi_l,
                             int d, int64_t chi_r, int dl, int dr) {
  const int64_t total = chi_l * d * chi_r;
  for (int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; idx < total;
       idx += int64_t(gridDim.x) * blockDim.x) {
    const int64_t a = idx / (d * chi_r);
    const int s = int((idx / chi_r) % d);
    const int64_t c = idx % chi_r;
    double acc = 0.0;
    for (int w = 0; w < dl; ++w) {
      const double lw = L[(a * dl + w) * chi_l + a];
      for (int v = 0; v < dr; ++v)
        acc = fma(lw * W[((w * dr + v) * d + s) * d + s], R[(c * dr + v) * chi_r + c], acc);
    }
    diag[idx] = acc;
  }
}

__global__ void full_matrix1_kernel(const double* __restrict__ L, const double* __restrict__ W,
                                    const double* __restrict__ R, double* __restrict__ H,
                                    int64_t chi_l, int d, int64_t chi_r, int dl, int dr) {
  const int64_t n = chi_l * d * chi_r;
  const int64_t total = n * n;
  for (int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; idx < total;
       idx += int64_t(gridDim.x) * blockDim.x) {
    const int64_t row = idx / n, col = idx % n;
    const int64_t a = row / (d * chi_r), c = row % chi_r;
    const int s = int((row / chi_r) % d);
    const int64_t ap = col / (d * chi_r), cp = col % chi_r;
    const int sp = int((col / chi_r) % d);
    double acc = 0.0;
    for (int w = 0; w < dl; ++w) {
      const double lw = L[(a * dl + w) * chi_l + ap];
      if (lw == 0.0) continue;
      for (int v = 0; v < dr; ++v)
        acc = fma(lw * W[((w * dr + v) * d + s) * d + sp], R[(c * dr + v) * chi_r + cp], acc);
    }
    H[idx] = acc;
  }
}
}  // namespace

}  // namespace tnx

using namespace tnx;

static int check_site(const void* L, const void* W, const void* R, int64_t chi_l, int64_t d,
                      int64_t chi_r, int64_t dl, int64_t dr) {
  TNX_CHECK_ARG(L && W && R, "null L/W/R pointer");
  TNX_CHECK_ARG(chi_l > 0 && d > 0 && chi_r > 0 && dl > 0 && dr > 0,
                "non-positive dimension (chi_l=%lld d=%lld chi_r=%lld dl=%lld dr=%lld)",
                (long long)chi_l, (long long)d, (long long)chi_r, (long long)dl, (long long)dr);
  TNX_CHECK_SHAPE(dl * d <= 64 && dr * d <= 64, "MPO bond too large: dl*d=%lld dr*d=%lld (max 64)",
                  (long long)(dl * d), (long long)(dr * d));
  return TNX_OK;
}

extern "C" {

size_t tnx_matvec1_workspace_bytes(int64_t chi_l, int64_t d, int64_t chi_r, int64_t dl, int64_t dr,
                                   int precision) {
  if (precision == TNX_BF16X3 && mixed_supported(chi_l, d, chi_r, dl, dr))
    return matvec1_bf16x3_scratch_bytes(chi_l, d, chi_r, dl, dr);
  const size_t t = 2 * align_up(size_t(matvec1_scratch_elems(chi_l, d, chi_r, dl, dr)) * sizeof(double));
  return precision == TNX_FP64 ? t : t + align_up(matvec1_oz_bytes(chi_l, d, chi_r, dl, dr));
}

int tnx_matvec1(const double* L, const double* W, const double* R, const double* x, double* y,
                int64_t chi_l, int64_t d, int64_t chi_r, int64_t dl, int64_t dr, int precision,
                void* workspace, size_t workspace_bytes, void* stream) {
  TNX_TRY(check_site(L, W, R, chi_l, d, chi_r, dl, dr));
  TNX_CHECK_ARG(x && y, "null x/y pointer");
  TNX_CHECK_ARG(precision >= TNX_FP64 && precision <= TNX_DF64, "unknown precision %d", precision);
  size_t need = tnx_matvec1_workspace_bytes(chi_l, d, chi_r, dl, dr, precision);
  if (workspace_bytes < need || (need && !workspace)) {
    set_error("tnx_matvec1: workspace %zu bytes < required %zu", workspace_bytes, need);
    return TNX_ERR_WORKSPACE;
  }
  cudaStream_t st = as_stream(stream);
  // sites with a bond below 16 (the chain ends) are too small for the tensor-core tiles and
  // always run the FP64 kernels
  if (precision == TNX_BF16X3 && mixed_supported(chi_l, d, chi_r, dl, dr))
    return matvec1_bf16x3(L, W, R, x, y, chi_l, d, chi_r, dl, dr, workspace, workspace_bytes, st);
  Arena ar(workspace, workspace_bytes);
  const int64_t ne = matvec1_scratch_elems(chi_l, d, chi_r, dl, dr);
  double* T1 = ar.take<double>(ne);
  double* T2 = ar.take<double>(ne);
  const size_t ozb = precision == TNX_DF64 ? matvec1_oz_bytes(chi_l, d, chi_r, dl, dr) : 0;
  void* oz = ozb ? static_cast<void*>(ar.take<char>(ozb)) : nullptr;
  return matvec1_f64(L, W, R, x, y, chi_l, d, chi_r, dl, dr, T1, T2, st, precision == TNX_DF64, oz, ozb);
}

int tnx_diag1(const double* L, const double* W, const double* R, double* diag, int64_t chi_l,
              int64_t d, int64_t chi_r, int64_t dl, int64_t dr, void* stream) {
  TNX_TRY(check_site(L, W, R, chi_l, d, chi_r, dl, dr));
  TNX_CHECK_ARG(diag, "null diag pointer");
  int64_t total = chi_l * d * chi_r;
  int64_t blocks = (total + 255) / 256;
  if (blocks > 152 * 16) blocks = 152 * 16;
  diag1_kernel<<<(unsigned)blocks, 256, 0, as_stream(stream)>>>(L, W, R, diag, chi_l, (int)d, chi_r,
                                                                (int)dl, (int)dr);
  TNX_LAUNCH_CHECK();
  return TNX_OK;
}

int tnx_full_matrix1(const double* L, const double* W, const double* R, double* H, int64_t chi_l,
                     int64_t d, int64_t chi_r, int64_t dl, int64_t dr, void* stream) {
  TNX_TRY(check_site(L, W, R, chi_l, d, chi_r, dl, dr));
  TNX_CHECK_ARG(H, "null H pointer");
  int64_t n = chi_l * d * chi_r;
  TNX_CHECK_SHAPE(n <= 8192, "dense effective Hamiltonian limited to 8192 rows (got %lld)", (long long)n);
  int64_t blocks = (n * n + 255) / 256;
  if (blocks > 152 * 16) blocks = 152 * 16;
  full_matrix1_kernel<<<(unsigned)blocks, 256, 0, as_stream(stream)>>>(L, W, R, H, chi_l, (int)d, chi_r,
                                                                       (int)dl, (int)dr);
  TNX_LAUNCH_CHECK();
  return TNX_OK;
}

// FP64-class scratch of the environment update's two GEMMs (tensor-core path)
static size_t env_oz_bytes(int direction, int64_t chi_l, int64_t d, int64_t chi_r, int64_t dl, int64_t dr) {
  int64_t g[2][3];
  if (direction == 1) {
    int64_t a[2][3] = {{dl * chi_l, d * chi_r, chi_l}, {chi_r * dr, chi_r, chi_l * d}};
    memcpy(g, a, sizeof(g));
  } else {
    int64_t a[2][3] = {{chi_l * d, dr * chi_r, chi_r}, {chi_l * dl, chi_l, d * chi_r}};
    memcpy(g, a, sizeof(g));
  }
  size_t out = 0;
  for (auto& x : g)
    if (use_oz(x[0], x[1], x[2])) {
      const size_t b = gemm_oz_workspace_bytes(x[0], x[1], x[2]);
      out = b > out ? b : out;
    }
  return out;
}

size_t tnx_env_update_workspace_bytes(int direction, int64_t chi_l, int64_t d, int64_t chi_r,
                                      int64_t dl, int64_t dr, int precision) {
  const size_t t = 2 * align_up(size_t(matvec1_scratch_elems(chi_l, d, chi_r, dl, dr)) * sizeof(double));
  if (!use_df64(precision)) return t;
  return t + align_up(env_oz_bytes(direction == -1 ? -1 : 1, chi_l, d, chi_r, dl, dr));
}

int tnx_env_update(int direction, const double* E_in, const double* A, const double* W,
                   double* E_out, int64_t chi_l, int64_t d, int64_t chi_r, int64_t dl, int64_t dr,
                   int precision, void* workspace, size_t workspace_bytes, void* stream) {
  TNX_TRY(check_site(E_in, W, A, chi_l, d, chi_r, dl, dr));
  TNX_CHECK_ARG(E_out, "null E_out pointer");
  TNX_CHECK_ARG(direction == 1 || direction == -1, "direction must be +1 or -1 (got %d)", direction);
  TNX_CHECK_ARG(precision >= TNX_FP64 && precision <= TNX_DF64, "unknown precision %d", precision);
  const bool df = use_df64(precision);
  size_t need = tnx_env_update_workspace_bytes(direction, chi_l, d, chi_r, dl, dr, precision);
  if (workspace_bytes < need || !workspace) {
    set_error("tnx_env_update: workspace %zu bytes < required %zu", workspace_bytes, need);
    return TNX_ERR_WORKSPACE;
  }
  cudaStream_t st = as_stream(stream);
  Arena ar(workspace, workspace_bytes);
  const int64_t ne = matvec1_scratch_elems(chi_l, d, chi_r, dl, dr);
  double* T1 = ar.take<double>(ne);
  double* T2 = ar.take<double>(ne);
  const size_t ozb = df ? env_oz_bytes(direction, chi_l, d, chi_r, dl, dr) : 0;
  void* oz = ozb ? static_cast<void*>(ar.take<char>(ozb)) : nullptr;
  if (direction == 1) {
    // T1[(w,a'),(s,c)] = sum_a L[a,(w,a')] A[a,(s,c)]
    TNX_TRY(gemm_fp64_class_oz(df, true, false, dl * chi_l, d * chi_r, chi_l, 1.0, E_in, dl * chi_l, A, d * chi_r,
                               0.0, T1, d * chi_r, oz, ozb, st));
    TNX_TRY(wcontract_left(T1, W, T2, chi_l, d, chi_r, dl, dr, st));
    // L'[(c,v),c'] = sum_{(a',s')} T2[(a',s'),(c,v)] A[(a',s'),c']
    TNX_TRY(gemm_fp64_class_oz(df, true, false, chi_r * dr, chi_r, chi_l * d, 1.0, T2, chi_r * dr, A, chi_r, 0.0,
                               E_out, chi_r, oz, ozb, st));
  } else {
    // T1[(a,s),(v,c')] = sum_c A[(a,s),c] R[c,(v,c')]
    TNX_TRY(gemm_fp64_class_oz(df, false, false, chi_l * d, dr * chi_r, chi_r, 1.0, A, chi_r, E_in, dr * chi_r,
                               0.0, T1, dr * chi_r, oz, ozb, st));
    TNX_TRY(wcontract_right(T1, W, T2, chi_l, d, chi_r, dl, dr, st));
    // R'[(a,w),a'] = sum_{(s',c')} T2[(a,w),(s',c')] A[a',(s',c')]
    TNX_TRY(gemm_fp64_class_oz(df, false, true, chi_l * dl, chi_l, d * chi_r, 1.0, T2, d * chi_r, A, d * chi_r,
                               0.0, E_out, chi_l, oz, ozb, st));
  }
  return TNX_OK;
}

int tnx_gemm_f64(int trans_a, int trans_b, int64_t m, int64_t n, int64_t k, double alpha,
                 const double* A, int64_t lda, int64_t stride_a, const double* B, int64_t ldb,
                 int64_t stride_b, double beta, double* C, int64_t ldc, int64_t stride_c,
                 int64_t batch, void* stream) {
  TNX_CHECK_ARG(A && B && C, "null pointer");
  TNX_CHECK_ARG(m >= 0 && n >= 0 && k >= 0 && batch >= 0, "negative size");
  return gemm_f64(trans_a != 0, trans_b != 0, m, n, k, alpha, A, lda, stride_a, B, ldb, stride_b, beta,
                  C, ldc, stride_c, batch, as_stream(stream));
}

}  // extern "C"
