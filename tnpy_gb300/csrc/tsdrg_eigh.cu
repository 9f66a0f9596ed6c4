// Lowest-k eigenpairs of tSDRG block Hamiltonians H = sum_w A_w (x) B_w without forming H.
//
// Reference: TreeTensorNetworkSDRG.block_eigen_solver (tnpy/tsdrg.py:569-592) diagonalises
// the dense two-block Hamiltonian of block_hamiltonian (:607-631) with np.linalg.eigh and keeps
// the lowest chi pairs. Here A_w = W1[0, w] (m1 x m1) and B_w = W2[w, dr2-1] (m2 x m2), so
// H v = sum_w vec(A_w X B_w^T) for X the m1 x m2 reshaping of v: a matvec costs
// 2 D m1 m2 (m1 + m2) flops instead of 2 (m1 m2)^2 and only the small factors sit in shared
// memory. One CTA per block, batched over blocks and disorder realisations:
//
//   1. kron_chfsi_kernel, FP32: Chebyshev-filtered subspace iteration on p = k + guard vectors:
//      Rayleigh-Ritz, a degree-10 Chebyshev filter damping [theta_p, upper bound] (from 24 Lanczos
//      steps: largest Ritz value + |beta|), CGS2; until the k wanted residuals reach FP32 rounding.
//   2a. FP64 precision, kron_polish_kernel: from those vectors, Rayleigh-Ritz, residuals,
//      convergence test and the vectors in FP64; only the correction of each vector,
//      e ~ -(H - theta_i)^-1 r_i in the complement of the subspace, is computed in FP32, by 48 steps
//      of the Chebyshev recurrence on the residual: with T_n(H) x = t_n x + d_n, the scaled
//      e_n = d_n / t_n obeys e_{n+1} = 2 q_n (H' e_n + r') - q_n q_{n-1} e_{n-1},
//      q_n = t_n / t_{n+1}, H' and r' in filter coordinates. A correction's relative error of
//      ~1e-5 only slows the outer iteration, whose end is the FP64 residual of 1e-13.
//   2b. FP64-class precisions, kron_refine_kernel: one FP64 Rayleigh-Ritz of the k FP32 vectors.
//      Ritz values are second order in the subspace error, so an FP32 subspace (~1e-6) gives
//      FP64-accurate kept spectra.
//
// What bounds it: an FP64 instruction holds its sub-partition's pipe for 64 clocks a warp. Ten FP64
// products per outer step, a one-warp FP64 Jacobi of the projected matrix (2.6 ms each) and a
// Gram-Schmidt with a warp reduction per pair took 92 ms for 16 blocks of m = 256, k = 16 and 2.0 s
// for 160 of m = 1024, k = 32 (both stages, per call). Now the filter runs in FP32 on the residual,
// one FP64 product is left per step, the projected problem is a whole CTA's (jacobi.cuh) and takes
// the vectors as they are (X^T X by Cholesky, no Gram-Schmidt), and a cluster of up to eight CTAs
// shares a block while the batch leaves SMs idle: 7.7 ms and 168 ms; 4 blocks of m = 1024 1139 and
// 19 ms. FP64-class precisions (FP32 stage and one Rayleigh-Ritz): 16 blocks 15.8 and 3.9 ms.
//
// A product runs one vector (two, for nodes of at most 16 states; four, where one has at most 8) per warp: the lane holds column
// b2 of X in registers, T = A_w X with A_w read as broadcast vectors, T is turned around through
// the warp's shared-memory tile, and the lane then holds row k1 of T and of the sum of T B_w^T. A
// whole filter runs in registers without touching memory in between.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "jacobi.cuh"
#include "tnx_internal.cuh"

namespace cg = cooperative_groups;

namespace tnx {
namespace {

constexpr int KT = 256;       // threads per CTA
constexpr int NW = KT / 32;
constexpr int KM1 = 32;       // largest node dimension (m1, m2)
constexpr int KP = 48;        // largest subspace block (k <= 32 kept + guard)
constexpr int KD = 6;         // largest MPO bond
constexpr int GL = KP + 1;    // row stride of the projected matrix
constexpr int TILE = KM1 * (KM1 + 1);  // one warp's tile
constexpr int GCH = 32;       // entries of a vector per step of the Gram product

template <typename T>
struct KSmall {
  T G[KP * GL];  // projected matrix (upper triangle); its eigenvectors as rows, stride KP, afterwards
  T V[KP * GL];  // rotations of small_eigh
  T theta[KP], scal[KP], red[NW];
  T cs[2][KP / 2], sn[2][KP / 2];
  int16_t sp[2][KP / 2], sq[2][KP / 2];
  int order[KP];
  int flag, any[2], rot;
  int ea[KD], eb[KD], eh;  // A_w is taken as A_w 2^-ea[w], B_w as B_w 2^-eb[w], H as H 2^-eh: eh = ea[w] + eb[w]
};

// A vector as the matrix that a product takes: nr rows (in registers) by nc columns (on lanes), entry (i, j) at
// i si + j sj. X itself, or X^T where that has the fewer columns.
struct Shape {
  int nr, nc, si, sj;
};
// operands of the products, padded with zeros to W x W: At[w][b1][k1] = A_w[k1][b1],
// Bt[w][b2][k2] = B_w[k2][b2]; W = 16 or 32 >= nr, nc (of X^T: B_w and A_w)
template <typename T>
struct Ops : Shape {
  const T *at, *bt;
  int D;
};
constexpr int ops_elems(int W, int D) { return 2 * D * W * W; }

// The CTAs of a block's cluster (one for large batches): vectors, entries and Gram chunks are dealt
// out over them, the p x p problems are solved by each.
struct Team {
  int rank, size;
  __device__ void sync() const {
    if (size > 1) cg::this_cluster().sync();
    else __syncthreads();
  }
};

template <typename T>
__device__ __forceinline__ T wsum(T v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// sum over the block, in every thread
template <typename T>
__device__ T bsum(T v, T* red) {
  v = wsum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  T t = T(0);
#pragma unroll
  for (int w = 0; w < NW; ++w) t += red[w];
  return t;
}

// largest eigenvalue of the symmetric tridiagonal (alpha[0..n), beta[1..n)) by Sturm bisection
__device__ double tridiag_max(const double* alpha, const double* beta, int n) {
  double lo = alpha[0], hi = alpha[0];
  for (int i = 0; i < n; ++i) {  // Gershgorin interval
    const double r = (i > 0 ? fabs(beta[i]) : 0.0) + (i + 1 < n ? fabs(beta[i + 1]) : 0.0);
    lo = fmin(lo, alpha[i] - r);
    hi = fmax(hi, alpha[i] + r);
  }
  for (int it = 0; it < 60; ++it) {
    const double x = 0.5 * (lo + hi);
    int below = 0;  // eigenvalues < x
    double q = alpha[0] - x;
    below += q < 0.0;
    for (int i = 1; i < n; ++i) {
      if (q == 0.0) q = 1e-300;
      q = alpha[i] - x - beta[i] * beta[i] / q;
      below += q < 0.0;
    }
    if (below == n) hi = x;  // every eigenvalue below x
    else lo = x;
  }
  return hi;
}

__device__ __forceinline__ void load4(const float* p, float (&o)[4]) {
  const float4 q = *reinterpret_cast<const float4*>(p);
  o[0] = q.x; o[1] = q.y; o[2] = q.z; o[3] = q.w;
}
__device__ __forceinline__ void load4(const double* p, double (&o)[4]) {
  const double2 q = *reinterpret_cast<const double2*>(p), r = *reinterpret_cast<const double2*>(p + 2);
  o[0] = q.x; o[1] = q.y; o[2] = r.x; o[3] = r.y;
}

// How a warp takes vectors: W rows in registers, L lanes a vector, 32 / L vectors at once
template <int W, int L>
__device__ __forceinline__ constexpr int tile_stride() { return W == L ? W * (W + 1) : W * L + 8; }

// y = sum A_w X B_w^T over w = w0, w0 + wstep, ... for the vector(s) of one warp; x[b1], y[k1] of column sl =
// lane mod L; tile: the vector's. With L = W the lane turns to row sl of T = A_w X for the second product and back at
// the end; with fewer lanes (L = 8) it stays with its column and reads T's rows from the tile. FULL runs over the
// padded W, so that all loads of a step are in flight together; otherwise the sums and rows stop at the
// dimensions, eight at a time. Padded to 32 x 32, a (24, 4) pair took over three times its operations, one vector a
// warp: 600 pairs, 32 kept, FP64-class 52 ms so and 17 ms with L = 8, FP64 245 and 61 ms; 200 of (17, 17) 34 and 21 ms with
// bounds; 32 x 32 in FP64 is 9 % faster padded, in FP32 2 % slower.
template <typename T, int W, int L, bool FULL>
__device__ __forceinline__ void warp_apply(const Ops<T>& o, const T (&x)[W], T (&y)[W], T* tile, int sl, int w0 = 0,
                                           int wstep = 1) {
  constexpr bool turn = W == L;
  constexpr int LT = turn ? W + 1 : L;  // row stride of the tile
  T acc[W];
#pragma unroll
  for (int i = 0; i < W; ++i) acc[i] = T(0);
  for (int w = w0; w < o.D; w += wstep) {
    const T* a = o.at + w * W * W;
#pragma unroll 1
    for (int k1 = 0; k1 < (FULL ? W : o.nr); k1 += 4) {
      T t[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll
      for (int b0 = 0; b0 < W; b0 += 8) {
        if (!FULL && b0 >= o.nr) continue;
#pragma unroll
        for (int b1 = b0; b1 < b0 + 8; ++b1) {
          T v[4];
          load4(a + b1 * W + k1, v);
#pragma unroll
          for (int i = 0; i < 4; ++i) t[i] = fma(v[i], x[b1], t[i]);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) tile[(k1 + i) * LT + sl] = t[i];
    }
    __syncwarp();
    const T* bm = o.bt + w * W * W;
    if constexpr (turn) {
#pragma unroll 2
      for (int b2 = 0; b2 < (FULL ? W : o.nc); ++b2) {
        const T tr = FULL || sl < o.nr ? tile[sl * LT + b2] : T(0);  // rows beyond were not written
#pragma unroll
        for (int k0 = 0; k0 < W; k0 += 8) {
          if (!FULL && k0 >= o.nc) continue;
#pragma unroll
          for (int k2 = k0; k2 < k0 + 8; k2 += 4) {
            T v[4];
            load4(bm + b2 * W + k2, v);
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[k2 + i] = fma(tr, v[i], acc[k2 + i]);
          }
        }
      }
    } else {
#pragma unroll
      for (int b0 = 0; b0 < L; b0 += 4) {
        if (b0 >= o.nc) continue;
        T b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) b[i] = bm[(b0 + i) * W + sl];
#pragma unroll
        for (int k0 = 0; k0 < W; k0 += 4) {
          if (k0 >= o.nr) continue;
#pragma unroll
          for (int k1 = k0; k1 < k0 + 4; ++k1) {
            T v[4];
            load4(tile + k1 * LT + b0, v);
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[k1] = fma(v[i], b[i], acc[k1]);
          }
        }
      }
    }
    __syncwarp();
  }
  if constexpr (turn) {
    // lane k1, entry k2 -> lane k2, entry k1
#pragma unroll
    for (int k2 = 0; k2 < W; ++k2) tile[sl * LT + k2] = acc[k2];
    __syncwarp();
#pragma unroll
    for (int k1 = 0; k1 < W; ++k1) y[k1] = tile[k1 * LT + sl];
    __syncwarp();
  } else {
#pragma unroll
    for (int k1 = 0; k1 < W; ++k1) y[k1] = acc[k1];
  }
}

// vector j of X (vector-major) into registers, column sl
template <typename T, int W, typename S>
__device__ __forceinline__ void load_vec(const S* X, int j, bool live, T (&x)[W], const Shape& o, int sl) {
#pragma unroll
  for (int i = 0; i < W; ++i)
    x[i] = (live && i < o.nr && sl < o.nc) ? T(X[size_t(j) * o.nr * o.nc + i * o.si + sl * o.sj]) : T(0);
}
template <typename T, int W>
__device__ __forceinline__ void store_vec(T* X, int j, bool live, const T (&x)[W], const Shape& o, int sl) {
#pragma unroll
  for (int i = 0; i < W; ++i)
    if (live && i < o.nr && sl < o.nc) X[size_t(j) * o.nr * o.nc + i * o.si + sl * o.sj] = x[i];
}

// f(j, live, sl, tile) for the vectors j < p, 32 / L per warp of the team; every
// lane of the warp calls it, live false past the end
template <typename T, int W, int L, typename F>
__device__ __forceinline__ void for_vectors(const Team& tm, int p, T* tiles, F f) {
  constexpr int PK = 32 / L;
  static_assert(PK * tile_stride<W, L>() <= TILE, "tiles of a warp's vectors");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane / L, sl = lane % L;
  T* tile = tiles + warp * TILE + sub * tile_stride<W, L>();
  for (int j0 = (warp * tm.size + tm.rank) * PK; j0 < p; j0 += NW * tm.size * PK) f(j0 + sub, j0 + sub < p, sl, tile);
}

// Y_j = H X_j for j < p
template <typename T, int W, int L, bool FULL>
__device__ void apply_block(const Team& tm, const Ops<T>& o, const T* X, T* Y, int p, T* tiles) {
  for_vectors<T, W, L>(tm, p, tiles, [&](int j, bool live, int sl, T* tile) {
    T x[W], y[W];
    load_vec<T, W>(X, j, live, x, o, sl);
    warp_apply<T, W, L, FULL>(o, x, y, tile, sl);
    store_vec<T, W>(Y, j, live, y, o, sl);
  });
  tm.sync();
}

// y = H x for one vector in shared memory, the terms w spread over the CTA's warps; part: NW x m
template <typename T, int W, int L, bool FULL>
__device__ void apply_one(const Ops<T>& o, const T* x, T* y, T* tiles, T* part) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, m = o.nr * o.nc, sl = lane % L;
  if (warp < o.D) {
    T xv[W], yv[W];
    load_vec<T, W>(x, 0, true, xv, o, sl);
    warp_apply<T, W, L, FULL>(o, xv, yv, tiles + warp * TILE + lane / L * tile_stride<W, L>(), sl, warp, NW);
    store_vec<T, W>(part, warp, lane < L, yv, o, sl);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < m; e += KT) {
    T t = T(0);
    for (int w = 0; w < o.D; ++w) t += part[w * m + e];  // D <= NW
    y[e] = t;
  }
  __syncthreads();
}

// s.G = (X^T Y + Y^T X) / 2, and with WITH_S s.V = X^T X, above and on the diagonal: each CTA of the
// team sums its chunks of GCH entries, the partial sums are added in rank order. buf: scratch of
// 2 KP (GCH + 1) + (WITH_S ? 2 : 1) KP KP values
template <typename T, bool WITH_S>
__device__ void gram(const Team& tm, KSmall<T>& s, const T* X, const T* Y, int p, int m, T* buf) {
  T* xs = buf;
  T* ys = buf + KP * (GCH + 1);
  T* pg = ys + KP * (GCH + 1);  // [KP][KP] x_i . y_j of this CTA's chunks
  T* ps = pg + KP * KP;         // x_i . x_j
  constexpr int R = KP / 16;
  const int ti = threadIdx.x / 16, tj = threadIdx.x % 16;
  T acc[R][R], acs[R][R];
#pragma unroll
  for (int a = 0; a < R; ++a)
#pragma unroll
    for (int b = 0; b < R; ++b) acc[a][b] = acs[a][b] = T(0);
  for (int e0 = tm.rank * GCH; e0 < m; e0 += tm.size * GCH) {
    for (int q = threadIdx.x; q < KP * GCH; q += KT) {
      const int i = q / GCH, e = q % GCH;
      const bool in = i < p && e0 + e < m;
      xs[i * (GCH + 1) + e] = in ? X[size_t(i) * m + e0 + e] : T(0);
      ys[i * (GCH + 1) + e] = in ? Y[size_t(i) * m + e0 + e] : T(0);
    }
    __syncthreads();
    auto products = [&](auto rr) {  // rr x rr entries a thread: p <= 16 rr
      constexpr int RR = decltype(rr)::value;
#pragma unroll 4
      for (int e = 0; e < GCH; ++e) {
        T x[RR], z[RR], y[RR];
#pragma unroll
        for (int a = 0; a < RR; ++a) {
          x[a] = xs[(ti + 16 * a) * (GCH + 1) + e];
          y[a] = ys[(tj + 16 * a) * (GCH + 1) + e];
          if (WITH_S) z[a] = xs[(tj + 16 * a) * (GCH + 1) + e];
        }
#pragma unroll
        for (int a = 0; a < RR; ++a)
#pragma unroll
          for (int b = 0; b < RR; ++b) {
            acc[a][b] = fma(x[a], y[b], acc[a][b]);
            if (WITH_S && a <= b) acs[a][b] = fma(x[a], z[b], acs[a][b]);  // blocks on and above the diagonal
          }
      }
    };
    if (p <= 16) products(std::integral_constant<int, 1>{});
    else if (p <= 32) products(std::integral_constant<int, 2>{});
    else products(std::integral_constant<int, 3>{});
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < R; ++a)
#pragma unroll
    for (int b = 0; b < R; ++b) {
      pg[(ti + 16 * a) * KP + tj + 16 * b] = acc[a][b];
      if (WITH_S) ps[(ti + 16 * a) * KP + tj + 16 * b] = acs[a][b];
    }
  tm.sync();
  for (int q = threadIdx.x; q < p * p; q += KT) {
    const int i = q / p, j = q % p;
    if (i > j) continue;
    T g = T(0), h = T(0), z = T(0);
    for (int r = 0; r < tm.size; ++r) {
      const T* rg = tm.size > 1 ? cg::this_cluster().map_shared_rank(pg, r) : pg;
      g += rg[i * KP + j];
      h += rg[j * KP + i];
      if (WITH_S) z += rg[KP * KP + i * KP + j];
    }
    s.G[i * GL + j] = T(0.5) * (g + h);
    if (WITH_S) s.V[i * GL + j] = z;
  }
  tm.sync();  // no CTA rewrites its partial sums while another still reads them
}

// Eigendecomposition of the symmetric n x n s.G (upper triangle; n <= KP) by the whole CTA: parallel
// cyclic Jacobi, angles of a round by one warp while the warps of the other sub-partitions apply
// the round before to V, then the 2 x 2 blocks above the diagonal by one thread each. Eigenvalues
// ascending in s.theta, the vectors as rows of s.G (stride KP).
template <typename T>
__device__ void small_eigh(KSmall<T>& s, int n) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  T* G = s.G;
  T fro = T(0);
  for (int e = tid; e < n * n; e += KT) {
    const int i = e / n, j = e % n;
    s.V[i * GL + j] = i == j ? T(1) : T(0);
    if (i <= j) fro += (i == j ? T(1) : T(2)) * G[i * GL + j] * G[i * GL + j];
  }
  fro = sqrt(bsum(fro, s.red));
  const T floor = (sizeof(T) == 4 ? T(1e-7) : T(2e-16)) * fro;
  const int np = n + (n & 1), npairs = np / 2;
  auto at = [&](int i, int j) -> T& { return i < j ? G[i * GL + j] : G[j * GL + i]; };
  auto update_v = [&](int u, int slot, int slots) {
    for (int l = slot; l < npairs; l += slots) {
      const T sn = s.sn[u][l];
      if (jac::bits(sn) == 0) continue;
      const T c = s.cs[u][l];
      const int p = s.sp[u][l], q = s.sq[u][l];
      for (int j = lane; j < n; j += 32) {
        const T vp = s.V[j * GL + p], vq = s.V[j * GL + q];
        s.V[j * GL + p] = fma(c, vp, -sn * vq);
        s.V[j * GL + q] = fma(sn, vp, c * vq);
      }
    }
  };
  bool pending = false;
  int u = 0;
  for (int sweep = 0; sweep < 40 && n > 1; ++sweep) {
    if (tid == 0) s.rot = 0;
    for (int r = 0; r < np - 1; ++r, u ^= 1) {
      if (warp == 0) {
        bool rot = false;
        if (lane < npairs) {
          int p, q;
          jac::pair_of(lane, r, np, p, q);
          T c = T(1), sn = T(0);
          if (q < n) {
            const T apq = G[p * GL + q];
            if (abs(apq) > floor) {
              T t;
              const T app = G[p * GL + p], aqq = G[q * GL + q];
              jac::angle(apq, aqq - app, t, c, sn);
              G[p * GL + p] = fma(-t, apq, app);
              G[q * GL + q] = fma(t, apq, aqq);
              G[p * GL + q] = T(0);
              rot = true;
            }
          }
          s.sp[u][lane] = int16_t(p);
          s.sq[u][lane] = int16_t(q);
          s.cs[u][lane] = c;
          s.sn[u][lane] = sn;
        }
        const bool any = __any_sync(0xffffffffu, rot);
        if (lane == 0) {
          s.any[u] = any;
          if (any) s.rot = 1;
        }
      } else if (pending && (warp & 3) != 0) {
        update_v(u ^ 1, warp - 1 - (warp >> 2), NW - NW / 4);
      }
      __syncthreads();
      pending = s.any[u];
      if (!pending) continue;
      for (int x = tid; x < (npairs + 1) / 2 * (npairs - 1); x += KT) {
        const int w = x / (npairs - 1), y = x % (npairs - 1), k2 = npairs - 1 - w, n1 = npairs - 1 - w;
        if (y >= n1 && k2 <= w) continue;  // the middle row of an odd number of pairs
        const int k = y < n1 ? w : k2, l = y < n1 ? w + 1 + y : k2 + 1 + (y - n1);
        const T sk = s.sn[u][k], sl = s.sn[u][l];
        if ((jac::bits(sk) | jac::bits(sl)) == 0) continue;
        const int pk = s.sp[u][k], qk = s.sq[u][k], pl = s.sp[u][l], ql = s.sq[u][l];
        const bool row2 = qk < n, col2 = ql < n;
        T a = at(pk, pl), b = col2 ? at(pk, ql) : T(0), c = row2 ? at(qk, pl) : T(0),
          d = row2 && col2 ? at(qk, ql) : T(0);
        if (jac::bits(sl)) {
          const T cc = s.cs[u][l], a0 = a, c0 = c;
          a = fma(cc, a0, -sl * b);
          b = fma(sl, a0, cc * b);
          c = fma(cc, c0, -sl * d);
          d = fma(sl, c0, cc * d);
        }
        if (jac::bits(sk)) {
          const T cc = s.cs[u][k], a0 = a, b0 = b;
          a = fma(cc, a0, -sk * c);
          c = fma(sk, a0, cc * c);
          b = fma(cc, b0, -sk * d);
          d = fma(sk, b0, cc * d);
        }
        at(pk, pl) = a;
        if (col2) at(pk, ql) = b;
        if (row2) at(qk, pl) = c;
        if (row2 && col2) at(qk, ql) = d;
      }
      __syncthreads();
    }
    const int rot = s.rot;
    __syncthreads();
    if (!rot) break;
  }
  if (pending) update_v(u ^ 1, warp, NW);
  if (tid < n) {
    const T di = G[tid * GL + tid];
    const auto ki = jac::sort_key(di);
    int rank = 0;  // by integer keys: order[] is complete also where G holds NaN
    for (int j = 0; j < n; ++j) {
      const auto kj = jac::sort_key(G[j * GL + j]);
      rank += (kj < ki) || (kj == ki && j < tid);
    }
    s.order[rank] = tid;
    s.theta[rank] = di;
  }
  __syncthreads();
  for (int e = tid; e < KP * n; e += KT) {  // rows padded with zeros to KP
    const int r = e / KP, i = e % KP;
    G[e] = i < n ? s.V[i * GL + s.order[r]] : T(0);
  }
  __syncthreads();
}

// X <- X Q: vector r = sum_i Q[r][i] X_i (Q = s.G, rows of stride KP), in place: each entry's row of all
// p vectors is one thread's
template <typename T>
__device__ void rotate(const Team& tm, const KSmall<T>& s, T* X, int p, int m) {
  for (int e = tm.rank * KT + threadIdx.x; e < m; e += tm.size * KT) {
    T x[KP];
#pragma unroll
    for (int i = 0; i < KP; ++i) x[i] = i < p ? X[size_t(i) * m + e] : T(0);
    auto products = [&](auto nn) {  // p <= N
      constexpr int N = decltype(nn)::value;
#pragma unroll 2
      for (int r = 0; r < p; ++r) {
        T t[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll
        for (int i = 0; i < N; i += 4) {
          T q[4];
          load4(s.G + r * KP + i, q);
#pragma unroll
          for (int h = 0; h < 4; ++h) t[h] = fma(x[i + h], q[h], t[h]);
        }
        X[size_t(r) * m + e] = (t[0] + t[1]) + (t[2] + t[3]);
      }
    };
    if (p <= 16) products(std::integral_constant<int, 16>{});
    else if (p <= 32) products(std::integral_constant<int, 32>{});
    else products(std::integral_constant<int, 48>{});
  }
}

// Rayleigh-Ritz of p vectors that are not orthonormal, from s.G = X^T H X and s.V = X^T X (upper
// triangles): S = U^T U, eigenpairs of U^-T G U^-1, and the rows of s.G become the columns of U^-1 Q.
// scr: 2 KP GL + KP values. False (in every thread) where S is not positive definite to working
// accuracy.
template <typename T>
__device__ bool small_eigh_general(KSmall<T>& s, int p, T* scr) {
  T* U = scr;              // [KP][GL]
  T* Z = scr + KP * GL;    // [KP][GL]
  T* rinv = Z + KP * GL;   // 1 / U_jj
  const int tid = threadIdx.x;
  for (int q = tid; q < p * p; q += KT) {
    const int i = q / p, j = q % p;
    U[i * GL + j] = i <= j ? s.V[i * GL + j] : T(0);
    Z[i * GL + j] = i <= j ? s.G[i * GL + j] : s.G[j * GL + i];
  }
  __syncthreads();
  bool ok = true;
  // right-looking: factor S and Z <- U^-T Z in one loop over the pivots
  for (int j = 0; j < p; ++j) {
    const T d = U[j * GL + j];
    ok = ok && d > T(1e-8);  // uniform: every thread reads the same pivot (vectors are near unit length)
    __syncthreads();
    for (int c = tid; c < 2 * p; c += KT) {
      const T r = ok ? jac::rsqrt_exact(d) : T(1);
      if (c == 0) rinv[j] = r;
      if (c < p) {
        if (c >= j) U[j * GL + c] *= r;
      } else {
        Z[j * GL + c - p] *= r;
      }
    }
    __syncthreads();
    const int rows = p - 1 - j;
    for (int q = tid; q < rows * p; q += KT) {
      const int i = j + 1 + q / p, c = q % p;
      const T f = U[j * GL + i];
      if (c >= i) U[i * GL + c] = fma(-f, U[j * GL + c], U[i * GL + c]);
      Z[i * GL + c] = fma(-f, Z[j * GL + c], Z[i * GL + c]);
    }
    __syncthreads();
  }
  if (!ok) return false;
  // Z <- Z U^-1, column by column
  for (int j = 0; j < p; ++j) {
    for (int i = tid; i < p; i += KT) Z[i * GL + j] *= rinv[j];
    __syncthreads();
    const int cols = p - 1 - j;
    for (int q = tid; q < cols * p; q += KT) {
      const int c = j + 1 + q / p, i = q % p;
      Z[i * GL + c] = fma(-Z[i * GL + j], U[j * GL + c], Z[i * GL + c]);
    }
    __syncthreads();
  }
  for (int q = tid; q < p * p; q += KT) {
    const int i = q / p, j = q % p;
    if (i <= j) s.G[i * GL + j] = T(0.5) * (Z[i * GL + j] + Z[j * GL + i]);
  }
  __syncthreads();
  small_eigh(s, p);
  // rows r of s.G are the eigenvectors q_r: solve U v = q_r for all of them, from the last entry up
  for (int j = p - 1; j >= 0; --j) {
    for (int r = tid; r < p; r += KT) s.G[r * KP + j] *= rinv[j];
    __syncthreads();
    for (int q = tid; q < j * p; q += KT) {
      const int r = q / j, i = q % j;
      s.G[r * KP + i] = fma(-U[i * GL + j], s.G[r * KP + j], s.G[r * KP + i]);
    }
    __syncthreads();
  }
  return true;
}

// CGS2 of the p vectors of X, in order; the second pass only where the first took more than half of
// a vector's squared norm (DGKS). xj: m values.
template <typename T>
__device__ void orthonormalise(KSmall<T>& s, T* X, int p, int m, T* xj) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int j = 0; j < p; ++j) {
    T* x = X + size_t(j) * m;
    T part = T(0);
    for (int e = threadIdx.x; e < m; e += KT) {
      const T v = x[e];
      xj[e] = v;
      part = fma(v, v, part);
    }
    T nrm = bsum(part, s.red);
    for (int pass = 0; pass < 2 && j > 0; ++pass) {
      __syncthreads();
      for (int i = warp; i < j; i += NW) {
        const T* xi = X + size_t(i) * m;
        T d = T(0);
        for (int e = lane; e < m; e += 32) d = fma(xi[e], xj[e], d);
        d = wsum(d);
        if (lane == 0) s.scal[i] = d;
      }
      __syncthreads();
      part = T(0);
      for (int e = threadIdx.x; e < m; e += KT) {
        T t = xj[e];
#pragma unroll 8
        for (int i = 0; i < j; ++i) t = fma(-s.scal[i], X[size_t(i) * m + e], t);
        xj[e] = t;
        part = fma(t, t, part);
      }
      const T after = bsum(part, s.red);
      const bool enough = after >= T(0.5) * nrm;
      nrm = after;
      if (enough) break;
    }
    const T inv = nrm > T(0) ? T(1) / sqrt(nrm) : T(0);
    for (int e = threadIdx.x; e < m; e += KT) x[e] = xj[e] * inv;
    __syncthreads();
  }
}

// deterministic pseudo-random start vectors in [-1, 1)
__device__ __forceinline__ float hash_unit(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t h = a * 0x9E3779B1u ^ (b + 0x7F4A7C15u) * 0x85EBCA77u ^ (c + 0x165667B1u) * 0xC2B2AE3Du;
  h ^= h >> 15;
  h *= 0x2C1B3C6Du;
  h ^= h >> 12;
  h *= 0x297A2D39u;
  h ^= h >> 15;
  return float(h) * (2.0f / 4294967296.0f) - 1.0f;
}

// Powers of two that bring H to the order of one, so that no Hamiltonian is out of FP32's range: the largest A_w
// (x) B_w, by its exponents, becomes one. Exact, and every step of the solvers is homogeneous in H. A term with a zero
// factor is dropped.
template <typename T>
__device__ void scale_ops(KSmall<T>& s, const double* W1, const double* W2, int m1, int m2, int dr2, int D) {
  auto field = [](double x) { return (__double2hiint(x) >> 20) & 0x7ff; };
  for (int i = threadIdx.x; i < KD; i += KT) s.ea[i] = s.eb[i] = 0;
  __syncthreads();
  for (int w = 0; w < D; ++w) {
    const double* a = W1 + size_t(w) * m1 * m1;  // row 0 of W1
    const double* b = W2 + (size_t(w) * dr2 + dr2 - 1) * m2 * m2;
    int xa = 0, xb = 0;
    for (int e = threadIdx.x; e < m1 * m1; e += KT) xa = max(xa, field(a[e]));
    for (int e = threadIdx.x; e < m2 * m2; e += KT) xb = max(xb, field(b[e]));
    xa = __reduce_max_sync(0xffffffffu, xa);
    xb = __reduce_max_sync(0xffffffffu, xb);
    if ((threadIdx.x & 31) == 0) {
      atomicMax(&s.ea[w], xa);
      atomicMax(&s.eb[w], xb);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int e = -5000;
    for (int w = 0; w < D; ++w)
      if (s.ea[w] && s.eb[w]) e = max(e, s.ea[w] + s.eb[w] - 2046);
    s.eh = e == -5000 ? 0 : e;
    for (int w = 0; w < D; ++w) {
      const bool zero = !s.ea[w] || !s.eb[w];
      s.ea[w] = zero ? 5000 : s.ea[w] - 1023;
      s.eb[w] = zero ? 5000 : s.eh - s.ea[w];
    }
  }
  __syncthreads();
}

// A_w = W1[0, w] and B_w = W2[w, dr2 - 1], scaled by scale_ops, as padded operands of type T; for X^T if
// `transposed`
template <typename T, int W, typename S>
__device__ Ops<T> load_ops(const KSmall<S>& s, const double* W1, const double* W2, int m1, int m2, int dr2, int D,
                           bool transposed, T* mem) {
  T* at = transposed ? mem + D * W * W : mem;
  T* bt = transposed ? mem : mem + D * W * W;
  for (int e = threadIdx.x; e < D * W * W; e += KT) {
    const int w = e / (W * W), b = e / W % W, k = e % W;
    const double x = (b < m1 && k < m1) ? W1[(size_t(w) * m1 + k) * m1 + b] : 0.0;  // row 0 of W1
    const double y = (b < m2 && k < m2) ? W2[((size_t(w) * dr2 + dr2 - 1) * m2 + k) * m2 + b] : 0.0;
    at[e] = jac::bits(x) == 0 ? T(0) : T(scale_pow2(x, -s.ea[w]));
    bt[e] = jac::bits(y) == 0 ? T(0) : T(scale_pow2(y, -s.eb[w]));
  }
  __syncthreads();
  const Shape sh = transposed ? Shape{m2, m1, 1, m2} : Shape{m1, m2, m2, 1};
  return {sh, mem, mem + D * W * W, D};
}

// Upper end of the spectrum for the filter: 24 Lanczos steps on one vector give the largest
// Ritz value theta_max; theta_max + |beta_last| (plus 1% of the Ritz range) bounds lambda_max
// in practice and is far tighter than the norm bound sum_w ||A_w||_inf ||B_w||_inf, which caps
// it. A tighter damping interval makes every filter application converge faster. mem: (NW + 3) m.
template <int W, int L, bool FULL>
__device__ float upper_bound(KSmall<float>& s, const Ops<float>& o, int b, float* tiles, float* mem) {
  __shared__ double lal[25], lbe[25];
  __shared__ unsigned norm[2 * KD];
  const int m = o.nr * o.nc, nl = m < 24 ? m : 24;
  if (threadIdx.x < 2 * KD) norm[threadIdx.x] = 0u;
  __syncthreads();
  for (int r = threadIdx.x; r < o.D * (o.nr + o.nc); r += KT) {  // row sums
    const bool a = r < o.D * o.nr;
    const int q = a ? r : r - o.D * o.nr, mm = a ? o.nr : o.nc, w = q / mm, k = q % mm;
    const float* x = (a ? o.at : o.bt) + w * W * W + k;
    float t = 0.f;
    for (int i = 0; i < mm; ++i) t += fabsf(x[i * W]);
    atomicMax(&norm[(a ? 0 : KD) + w], __float_as_uint(t));  // non-negative: ordered as integers
  }
  float* v = mem;
  float* vp = mem + m;
  float* w = mem + 2 * m;
  float* part = mem + 3 * m;
  float nv = 0.f;
  for (int e = threadIdx.x; e < m; e += KT) {
    v[e] = hash_unit(b + 7919u, 0u, uint32_t(e));
    vp[e] = 0.f;
    nv = fmaf(v[e], v[e], nv);
  }
  nv = sqrtf(bsum(nv, s.red));
  for (int e = threadIdx.x; e < m; e += KT) v[e] /= nv;
  __syncthreads();
  float beta = 0.f;
  int steps = 0;
  for (int j = 0; j < nl; ++j) {
    apply_one<float, W, L, FULL>(o, v, w, tiles, part);
    float t = 0.f;
    for (int e = threadIdx.x; e < m; e += KT) t = fmaf(w[e], v[e], t);
    const float alpha = bsum(t, s.red);
    t = 0.f;
    for (int e = threadIdx.x; e < m; e += KT) {
      w[e] -= alpha * v[e] + beta * vp[e];
      t = fmaf(w[e], w[e], t);
    }
    const float bnew = sqrtf(bsum(t, s.red));
    if (threadIdx.x == 0) {
      lal[j] = double(alpha);
      lbe[j + 1] = double(bnew);
    }
    steps = j + 1;
    if (!(bnew > 1e-12f * (fabsf(alpha) + 1e-30f))) break;
    for (int e = threadIdx.x; e < m; e += KT) {
      vp[e] = v[e];
      v[e] = w[e] / bnew;
    }
    beta = bnew;
    __syncthreads();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    lbe[0] = 0.0;
    double tmin = lal[0];
    for (int i = 0; i < steps; ++i) tmin = fmin(tmin, lal[i]);
    const double top = tridiag_max(lal, lbe, steps);
    double cap = 0.0;
    for (int w = 0; w < o.D; ++w) cap += double(__uint_as_float(norm[w])) * double(__uint_as_float(norm[KD + w]));
    const double est = top + fabs(lbe[steps]) + 0.01 * fabs(top - tmin) + 1e-12 * fabs(top);
    cap *= 1.01;
    s.scal[0] = float(est < cap ? est : cap);
  }
  __syncthreads();
  const float ub = s.scal[0] + 1e-30f;
  __syncthreads();
  return ub;
}

// scratch after the operands: the warps' tiles, the Gram buffers and partial sums, the matrices of
// small_eigh_general, one vector of orthonormalise (never at once), then the Lanczos vectors
template <typename T>
__host__ __device__ constexpr size_t scratch_elems(int max_m, bool lanczos) {
  size_t e = size_t(NW) * TILE;
  const size_t g = size_t(2) * KP * (GCH + 1) + 2 * KP * KP;
  e = g > e ? g : e;
  return e + (lanczos ? size_t(NW + 3) * max_m : 0);
}
static_assert(2 * KP * GL + KP <= NW * TILE && KM1 * KM1 <= NW * TILE, "scratch of the small problems");

// FP32 subspace iteration; `nout` of the Ritz vectors go to `out` (FP64, vector-major) and the filter's
// upper bound (of the scaled H) to bound[b].
template <int W, int L>
__device__ void chfsi(const Team& tm, const double* W1, const double* W2, int m1, int m2, int dr2, int k, int p, int D,
                      int b, float* X, float* Y, int max_outer, int degree, double* out, int nout, float* bound,
                      int* iters, unsigned char* raw) {
  constexpr bool FULL = W == 16;
  KSmall<float>& s = *reinterpret_cast<KSmall<float>*>(raw);
  float* mem = reinterpret_cast<float*>(raw + (sizeof(KSmall<float>) + 15) / 16 * 16);
  const int m = m1 * m2;
  scale_ops(s, W1, W2, m1, m2, dr2, D);
  const Ops<float> o = load_ops<float, W>(s, W1, W2, m1, m2, dr2, D, L < W && m1 < m2, mem);
  float* tiles = mem + ops_elems(W, D);
  const float ub = upper_bound<W, L, FULL>(s, o, b, tiles, tiles + scratch_elems<float>(0, false));
  auto orthonormal = [&] {  // one vector after the other: the first CTA's
    if (tm.rank == 0) orthonormalise(s, X, p, m, tiles);
    tm.sync();
  };
  if (tm.rank == 0)
    for (int e = threadIdx.x; e < p * m; e += KT) X[e] = hash_unit(b, e / m, e % m);
  __syncthreads();
  orthonormal();
  int it = 0;
  for (; it < max_outer; ++it) {
    // Rayleigh-Ritz: Y = H X, G = X^T Y
    apply_block<float, W, L, FULL>(tm, o, X, Y, p, tiles);
    gram<float, false>(tm, s, X, Y, p, m, tiles);
    small_eigh(s, p);
    rotate(tm, s, X, p, m);
    rotate(tm, s, Y, p, m);
    tm.sync();
    // residuals of the k wanted pairs: ||H x_i - theta_i x_i||
    const float scale = fmaxf(fabsf(s.theta[0]), fabsf(s.theta[p - 1]));
    if (threadIdx.x == 0) s.flag = 1;
    __syncthreads();
    for (int i = threadIdx.x >> 5; i < k; i += NW) {
      float part = 0.f;
      for (int e = threadIdx.x & 31; e < m; e += 32) {
        const float r = Y[size_t(i) * m + e] - s.theta[i] * X[size_t(i) * m + e];
        part = fmaf(r, r, part);
      }
      part = wsum(part);
      if ((threadIdx.x & 31) == 0 && !(sqrtf(part) <= 3e-6f * (scale + 1e-30f))) s.flag = 0;
    }
    __syncthreads();
    if (s.flag) break;
    tm.sync();  // every CTA has its residuals before the filter rewrites X
    // Chebyshev filter of degree `degree` on [a, ub], a = largest Ritz value of the block
    const float a = s.theta[p - 1];
    const float c = 0.5f * (a + ub), h = 0.5f * (ub - a) + 1e-30f;
    for_vectors<float, W, L>(tm, p, tiles, [&](int j, bool live, int sl, float* tile) {
      float prev[W], cur[W], hx[W];
      load_vec<float, W>(X, j, live, prev, o, sl);
      load_vec<float, W>(Y, j, live, cur, o, sl);
#pragma unroll
      for (int i = 0; i < W; ++i) cur[i] = (cur[i] - c * prev[i]) / h;
      for (int d = 2; d <= degree; ++d) {
        warp_apply<float, W, L, FULL>(o, cur, hx, tile, sl);
#pragma unroll
        for (int i = 0; i < W; ++i) {
          const float t = 2.f * (hx[i] - c * cur[i]) / h - prev[i];
          prev[i] = cur[i];
          cur[i] = t;
        }
      }
      store_vec<float, W>(X, j, live, cur, o, sl);
    });
    tm.sync();
    orthonormal();
  }
  for (int e = tm.rank * KT + threadIdx.x; e < nout * m; e += tm.size * KT) out[e] = double(X[e]);
  // iterations used, or -max_outer when the wanted residuals never reached the tolerance
  if (threadIdx.x == 0 && tm.rank == 0) {
    if (iters) iters[b] = s.flag ? it + 1 : -max_outer;
    if (bound) bound[b] = ub;
  }
  tm.sync();  // shared memory stays until no CTA reads it
}

// Where one node has more than 16 states, the lanes a vector takes while the other has no more
constexpr int NARROW = 8;

// meta[5b..5b+4] = m1, m2, dr2, k, p; the k Ritz vectors go to vec_base, all p when keep_guards
__global__ void __launch_bounds__(KT) kron_chfsi_kernel(const double* const* __restrict__ w1s,
                                                       const double* const* __restrict__ w2s,
                                                       const int* __restrict__ meta, int D, float* __restrict__ work,
                                                       int64_t work_stride, int max_outer, int degree,
                                                       double* __restrict__ vec_base, int64_t vec_stride,
                                                       int keep_guards, float* __restrict__ bounds,
                                                       int* __restrict__ out_iters, int team) {
  extern __shared__ __align__(16) unsigned char ksm_raw[];
  const Team tm{int(blockIdx.x % team), team};
  const int b = blockIdx.x / team;
  const int m1 = meta[5 * b], m2 = meta[5 * b + 1], dr2 = meta[5 * b + 2], k = meta[5 * b + 3], p = meta[5 * b + 4];
  float* X = work + size_t(b) * work_stride;
  float* Y = X + size_t(p) * m1 * m2;
  double* out = vec_base + size_t(b) * vec_stride;
  const int nout = keep_guards ? p : k;
  if (m1 <= 16 && m2 <= 16)
    chfsi<16, 16>(tm, w1s[b], w2s[b], m1, m2, dr2, k, p, D, b, X, Y, max_outer, degree, out, nout, bounds, out_iters,
                  ksm_raw);
  else if (min(m1, m2) <= NARROW)
    chfsi<32, NARROW>(tm, w1s[b], w2s[b], m1, m2, dr2, k, p, D, b, X, Y, max_outer, degree, out, nout, bounds, out_iters,
                      ksm_raw);
  else
    chfsi<32, 32>(tm, w1s[b], w2s[b], m1, m2, dr2, k, p, D, b, X, Y, max_outer, degree, out, nout, bounds, out_iters,
                  ksm_raw);
}

// e -= XF (XF^T e) for two vectors per group of L lanes
template <int W, int L>
__device__ __forceinline__ void project_out(const float* XF, int p, const Shape& o, int sl, float (&e)[W],
                                            float (&f)[W]) {
  for (int i = 0; i < p; ++i) {
    float x[W];
    load_vec<float, W>(XF, i, true, x, o, sl);
    float d = 0.f, g = 0.f;
#pragma unroll
    for (int q = 0; q < W; ++q) {
      d = fmaf(x[q], e[q], d);
      g = fmaf(x[q], f[q], g);
    }
#pragma unroll
    for (int q = L / 2; q > 0; q >>= 1) {
      d += __shfl_xor_sync(0xffffffffu, d, q);
      g += __shfl_xor_sync(0xffffffffu, g, q);
    }
#pragma unroll
    for (int q = 0; q < W; ++q) {
      e[q] = fmaf(-d, x[q], e[q]);
      f[q] = fmaf(-g, x[q], f[q]);
    }
  }
}

constexpr int POLISH_STEPS = 48;  // Chebyshev steps of a correction
constexpr int POLISH_PROJECT = 8;  // steps between projections onto the complement

// FP64 eigenpairs from the FP32 subspace in X (p vectors, vector-major): see the head of the file
template <int W, int L, bool FULL>
__device__ void polish(const Team& tm, const double* W1, const double* W2, int m1, int m2, int dr2, int k, int p,
                       int D, int b, double* X, double* Y, float* XF, float ub, int max_outer, double* ev, double* out,
                       int keep, int* iters, unsigned char* raw) {
  KSmall<double>& s = *reinterpret_cast<KSmall<double>*>(raw);
  double* mem = reinterpret_cast<double*>(raw + (sizeof(KSmall<double>) + 15) / 16 * 16);
  const int m = m1 * m2;
  scale_ops(s, W1, W2, m1, m2, dr2, D);
  const bool transposed = L < W && m1 < m2;
  const Ops<double> o = load_ops<double, W>(s, W1, W2, m1, m2, dr2, D, transposed, mem);
  double* tiles = mem + ops_elems(W, D);
  float* fmem = reinterpret_cast<float*>(tiles);  // FP32 operands and tiles of the corrections
  int it = 0;
  for (; it < max_outer; ++it) {
    apply_block<double, W, L, FULL>(tm, o, X, Y, p, tiles);
    gram<double, true>(tm, s, X, Y, p, m, tiles);
    if (!small_eigh_general(s, p, tiles)) {  // nearly dependent vectors: orthonormalise them first
      if (tm.rank == 0) orthonormalise(s, X, p, m, tiles);
      tm.sync();
      apply_block<double, W, L, FULL>(tm, o, X, Y, p, tiles);
      gram<double, false>(tm, s, X, Y, p, m, tiles);
      small_eigh(s, p);
    }
    rotate(tm, s, X, p, m);
    rotate(tm, s, Y, p, m);
    tm.sync();
    const double scale = fmax(fabs(s.theta[0]), fabs(s.theta[p - 1])) + 1e-30;
    if (threadIdx.x == 0) s.flag = 1;
    __syncthreads();
    // each CTA decides from all residuals; the FP32 copy of X is shared
    for (int i = threadIdx.x >> 5; i < p; i += NW) {
      double part = 0.0;
      for (int e = threadIdx.x & 31; e < m; e += 32) {
        const double x = X[size_t(i) * m + e], r = fma(-s.theta[i], x, Y[size_t(i) * m + e]);
        if (i % tm.size == tm.rank) XF[size_t(i) * m + e] = float(x);
        part = fma(r, r, part);
      }
      part = sqrt(wsum(part));
      if ((threadIdx.x & 31) == 0) {
        s.scal[i] = part;
        if (i < k && !(part <= 1e-13 * scale)) s.flag = 0;
      }
    }
    __syncthreads();
    if (s.flag) break;
    tm.sync();
    const double a = s.theta[p - 1], c = 0.5 * (a + double(ub)), h = 0.5 * (double(ub) - a) + 1e-30;
    const Ops<float> of = load_ops<float, W>(s, W1, W2, m1, m2, dr2, D, transposed, fmem);
    float* ftiles = fmem + ops_elems(W, D);
    const float cf = float(c), ih = float(1.0 / h);
    for_vectors<float, W, L>(tm, p, ftiles, [&](int j, bool live, int sl, float* tile) {
      const double th = live ? s.theta[j] : 0.0, nr = live ? s.scal[j] : 0.0;
      const bool work = nr > 0.0;
      const double inv = work ? 1.0 / (nr * h) : 0.0;
      float r[W], e[W], prev[W], hx[W];
#pragma unroll
      for (int i = 0; i < W; ++i) {
        r[i] = 0.f;
        if (work && i < o.nr && sl < o.nc) {
          const size_t q = size_t(j) * m + i * o.si + sl * o.sj;
          r[i] = float(fma(-th, X[q], Y[q]) * inv);
        }
      }
      const float tc = work ? float((th - c) / h) : -1.f;
      float q0 = 1.f / tc;
#pragma unroll
      for (int i = 0; i < W; ++i) {
        prev[i] = 0.f;
        e[i] = q0 * r[i];
      }
      for (int n = 1; n < POLISH_STEPS; ++n) {
        const float q1 = 1.f / (2.f * tc - q0);
        warp_apply<float, W, L, FULL>(of, e, hx, tile, sl);
#pragma unroll
        for (int i = 0; i < W; ++i) {
          const float t = 2.f * q1 * (fmaf(-cf, e[i], hx[i]) * ih + r[i]) - q1 * q0 * prev[i];
          prev[i] = e[i];
          e[i] = t;
        }
        q0 = q1;
        if ((n + 1) % POLISH_PROJECT == 0) project_out<W, L>(XF, p, o, sl, e, prev);
      }
      bool finite = true;
#pragma unroll
      for (int i = 0; i < W; ++i) finite = finite && fabsf(e[i]) < 1e30f;
      const unsigned group = (L == 32 ? ~0u : (1u << (L & 31)) - 1) << (((threadIdx.x & 31) / L) * L);
      finite = (__ballot_sync(0xffffffffu, finite) & group) == group;
      // x + |r| e, scaled to unit length (e is orthogonal to x)
      double len = 0.0;
      if (work && finite) {
#pragma unroll
        for (int i = 0; i < W; ++i) len = fma(nr * double(e[i]), nr * double(e[i]), len);
      }
#pragma unroll
      for (int q = L / 2; q > 0; q >>= 1) len += __shfl_xor_sync(0xffffffffu, len, q);
      if (work && finite) {
        const double f = 1.0 / sqrt(1.0 + len);
#pragma unroll
        for (int i = 0; i < W; ++i)
          if (i < o.nr && sl < o.nc) {
            const size_t q = size_t(j) * m + i * o.si + sl * o.sj;
            X[q] = fma(nr, double(e[i]), X[q]) * f;
          }
      }
    });
    tm.sync();
  }
  if (tm.rank == 0) {
    if (threadIdx.x < k) ev[threadIdx.x] = scale_pow2(s.theta[threadIdx.x], s.eh);
    for (int e = threadIdx.x; e < k * m; e += KT) {
      const int row = e / k, i = e % k;
      out[size_t(row) * keep + i] = X[size_t(i) * m + row];
    }
    if (threadIdx.x == 0 && iters) iters[b] = s.flag ? it + 1 : -max_outer;
  }
  tm.sync();  // shared memory stays until no CTA reads it
}

__global__ void __launch_bounds__(KT) kron_polish_kernel(const double* const* __restrict__ w1s,
                                                        const double* const* __restrict__ w2s,
                                                        const int* __restrict__ meta, int D, double* __restrict__ work,
                                                        int64_t work_stride, const float* __restrict__ bounds,
                                                        int max_outer, double* __restrict__ evals, int keep,
                                                        double* __restrict__ evecs, int max_m,
                                                        int* __restrict__ out_iters, int team) {
  extern __shared__ __align__(16) unsigned char ksm_raw[];
  const Team tm{int(blockIdx.x % team), team};
  const int b = blockIdx.x / team;
  const int m1 = meta[5 * b], m2 = meta[5 * b + 1], dr2 = meta[5 * b + 2], k = meta[5 * b + 3], p = meta[5 * b + 4];
  const size_t pm = size_t(p) * m1 * m2;
  double* X = work + size_t(b) * work_stride;
  double* Y = X + pm;
  float* XF = reinterpret_cast<float*>(Y + pm);
  double* ev = evals + size_t(b) * keep;
  double* out = evecs + size_t(b) * max_m * keep;  // [max_m][keep], like tnx_eigh_batched
  if (m1 <= 16 && m2 <= 16)
    polish<16, 16, true>(tm, w1s[b], w2s[b], m1, m2, dr2, k, p, D, b, X, Y, XF, bounds[b], max_outer, ev, out,
                        keep, out_iters, ksm_raw);
  else if (min(m1, m2) <= NARROW)
    polish<32, NARROW, false>(tm, w1s[b], w2s[b], m1, m2, dr2, k, p, D, b, X, Y, XF, bounds[b], max_outer, ev, out,
                             keep, out_iters, ksm_raw);
  else if (m1 > 24 && m2 > 24)
    polish<32, 32, true>(tm, w1s[b], w2s[b], m1, m2, dr2, k, p, D, b, X, Y, XF, bounds[b], max_outer, ev, out,
                        keep, out_iters, ksm_raw);
  else
    polish<32, 32, false>(tm, w1s[b], w2s[b], m1, m2, dr2, k, p, D, b, X, Y, XF, bounds[b], max_outer, ev, out,
                         keep, out_iters, ksm_raw);
}

template <int W, int L>
__device__ void ritz64(const Team& tm, KSmall<double>& s, const double* W1, const double* W2, int m1, int m2, int dr2,
                       int k, int D, double* V, double* Z, double* mem) {
  const int m = m1 * m2;
  scale_ops(s, W1, W2, m1, m2, dr2, D);
  const Ops<double> o = load_ops<double, W>(s, W1, W2, m1, m2, dr2, D, L < W && m1 < m2, mem);
  double* tiles = mem + ops_elems(W, D);
  orthonormalise(s, V, k, m, tiles);
  apply_block<double, W, L, W == 16>(tm, o, V, Z, k, tiles);
  gram<double, false>(tm, s, V, Z, k, m, tiles);
  small_eigh(s, k);
  rotate(tm, s, V, k, m);
  __syncthreads();
}

// FP64 Rayleigh-Ritz of the k vectors in vecs[b] (vector-major [k][m]); writes evals[b][i]
// ascending and evecs[b] as [m][k] (row-major, columns = eigenvectors); scratch: k m doubles.
__global__ void __launch_bounds__(KT) kron_refine_kernel(const double* const* __restrict__ w1s,
                                                        const double* const* __restrict__ w2s,
                                                        const int* __restrict__ meta, int D,
                                                        double* __restrict__ vec_base, int64_t vec_stride,
                                                        double* __restrict__ scratch, int64_t scratch_stride,
                                                        double* __restrict__ evals, int keep, double* __restrict__ evecs,
                                                        int max_m) {
  extern __shared__ __align__(16) unsigned char ksm_raw[];
  KSmall<double>& s = *reinterpret_cast<KSmall<double>*>(ksm_raw);
  double* mem = reinterpret_cast<double*>(ksm_raw + (sizeof(KSmall<double>) + 15) / 16 * 16);
  const int b = blockIdx.x;
  const int m1 = meta[5 * b], m2 = meta[5 * b + 1], dr2 = meta[5 * b + 2], k = meta[5 * b + 3];
  const int m = m1 * m2;
  double* V = vec_base + size_t(b) * vec_stride;
  double* Zb = scratch + size_t(b) * scratch_stride;
  const Team tm{0, 1};
  if (m1 <= 16 && m2 <= 16)
    ritz64<16, 16>(tm, s, w1s[b], w2s[b], m1, m2, dr2, k, D, V, Zb, mem);
  else if (min(m1, m2) <= NARROW)
    ritz64<32, NARROW>(tm, s, w1s[b], w2s[b], m1, m2, dr2, k, D, V, Zb, mem);
  else
    ritz64<32, 32>(tm, s, w1s[b], w2s[b], m1, m2, dr2, k, D, V, Zb, mem);
  double* ev = evals + size_t(b) * keep;
  for (int i = threadIdx.x; i < k; i += KT) ev[i] = scale_pow2(s.theta[i], s.eh);
  double* out = evecs + size_t(b) * max_m * keep;  // [max_m][keep], like tnx_eigh_batched
  for (int e = threadIdx.x; e < k * m; e += KT) {
    const int row = e / k, i = e % k;
    out[size_t(row) * keep + i] = V[size_t(i) * m + row];
  }
}

template <typename T>
size_t kron_smem(int D, int max_m, bool lanczos) {
  return (sizeof(KSmall<T>) + 15) / 16 * 16 + sizeof(T) * (ops_elems(KM1, D) + scratch_elems<T>(max_m, lanczos));
}
// the FP32 operands and tiles of the corrections take the place of the FP64 tiles and beyond
size_t polish_smem(int D) {
  const size_t f32 = sizeof(float) * (size_t(ops_elems(KM1, D)) + size_t(NW) * TILE),
               f64 = sizeof(double) * scratch_elems<double>(0, false);
  return (sizeof(KSmall<double>) + 15) / 16 * 16 + sizeof(double) * ops_elems(KM1, D) + (f32 > f64 ? f32 : f64);
}

// CTAs per block: a cluster of up to 8 while the batch leaves SMs idle
int team_for(int batch) {
  int t = 8;
  while (t > 1 && batch * t > 152) t /= 2;
  return t;
}

template <typename... P, typename... A>
int launch_team(void (*kernel)(P...), int batch, int team, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = unsigned(team);
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(unsigned(batch) * unsigned(team));
  cfg.blockDim = dim3(KT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = team > 1 ? 1 : 0;
  TNX_CUDA(cudaLaunchKernelEx(&cfg, kernel, P(args)...));
  TNX_LAUNCH_CHECK();
  return TNX_OK;
}

}  // namespace
}  // namespace tnx

using namespace tnx;

extern "C" {

size_t tnx_tsdrg_block_eigh_workspace_bytes(int batch, int max_m, int keep, int precision) {
  const size_t tsize = precision == TNX_FP64 ? 8 : 4;
  const size_t per_work = align_up(4 * size_t(KP) * max_m * tsize);
  const size_t per_vec = align_up(size_t(keep) * max_m * 8);
  const size_t per_scr = align_up(2 * size_t(keep) * max_m * 8);
  return size_t(batch) * (per_work + per_vec + per_scr) + 1024;
}

int tnx_tsdrg_block_eigh(const double* const* w1, const double* const* w2, const int* meta, int D, int batch,
                         int max_m, int keep, int precision, double* evals, double* evecs, int* iters,
                         void* workspace, size_t workspace_bytes, void* stream) {
  TNX_CHECK_ARG(w1 && w2 && meta && evals && evecs && workspace, "null pointer");
  TNX_CHECK_ARG(batch >= 0 && D > 0 && D <= KD && keep > 0 && keep <= 32, "bad batch / D / keep");
  TNX_CHECK_ARG(precision >= TNX_FP64 && precision <= TNX_DF64, "unknown precision %d", precision);
  TNX_CHECK_SHAPE(max_m > 0 && max_m <= KM1 * KM1, "block dimension %d outside (0, %d]", max_m, KM1 * KM1);
  if (batch == 0) return TNX_OK;
  const size_t need = tnx_tsdrg_block_eigh_workspace_bytes(batch, max_m, keep, precision);
  if (workspace_bytes < need) {
    set_error("tnx_tsdrg_block_eigh: workspace %zu bytes < required %zu", workspace_bytes, need);
    return TNX_ERR_WORKSPACE;
  }
  cudaStream_t st = as_stream(stream);
  const bool fp64 = precision == TNX_FP64;
  const size_t tsize = fp64 ? 8 : 4;
  const size_t per_work = align_up(4 * size_t(KP) * max_m * tsize);
  const size_t per_vec = align_up(size_t(keep) * max_m * 8);
  const size_t per_scr = align_up(2 * size_t(keep) * max_m * 8);
  char* base = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(workspace) + 255) & ~uintptr_t(255));
  char* work = base;
  double* vecs = reinterpret_cast<double*>(work + size_t(batch) * per_work);
  double* scr = reinterpret_cast<double*>(reinterpret_cast<char*>(vecs) + size_t(batch) * per_vec);
  const int max_outer = 60, degree = 10;
  static DeviceSet allowed_c, allowed_p, allowed_r;
  TNX_CUDA(allow_smem(kron_chfsi_kernel, kron_smem<float>(KD, KM1 * KM1, true), allowed_c));
  const int team = team_for(batch);
  const size_t smem_c = kron_smem<float>(D, max_m, true);
  profile_mark(KF_EIGH, st, true);
  if (fp64) {
    // the FP32 stage leaves all p vectors where the FP64 stage reads them (the first of work's four
    // blocks of p m doubles); its own two FP32 blocks are the last of the four
    TNX_CUDA(allow_smem(kron_polish_kernel, polish_smem(KD), allowed_p));
    float* bounds = reinterpret_cast<float*>(scr);
    float* w32 = reinterpret_cast<float*>(work) + 6 * size_t(KP) * max_m;
    double* w64 = reinterpret_cast<double*>(work);
    TNX_TRY(launch_team(kron_chfsi_kernel, batch, team, smem_c, st, w1, w2, meta, D, w32, int64_t(per_work / 4),
                        max_outer, degree, w64, int64_t(per_work / 8), 1, bounds, static_cast<int*>(nullptr), team));
    TNX_TRY(launch_team(kron_polish_kernel, batch, team, polish_smem(D), st, w1, w2, meta, D, w64,
                        int64_t(per_work / 8), bounds, max_outer, evals, keep, evecs, max_m, iters, team));
  } else {
    TNX_TRY(launch_team(kron_chfsi_kernel, batch, team, smem_c, st, w1, w2, meta, D, reinterpret_cast<float*>(work),
                        int64_t(per_work / 4), max_outer, degree, vecs, int64_t(per_vec / 8), 0,
                        static_cast<float*>(nullptr), iters, team));
    TNX_CUDA(allow_smem(kron_refine_kernel, kron_smem<double>(KD, KM1 * KM1, false), allowed_r));
    kron_refine_kernel<<<batch, KT, kron_smem<double>(D, max_m, false), st>>>(
        w1, w2, meta, D, vecs, int64_t(per_vec / 8), scr, int64_t(per_scr / 8), evals, keep, evecs, max_m);
    TNX_LAUNCH_CHECK();
  }
  profile_mark(KF_EIGH, st, false);
  return TNX_OK;
}

}  // extern "C"
