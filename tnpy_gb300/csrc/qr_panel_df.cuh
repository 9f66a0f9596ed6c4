// Double-FP32 cluster panel of the Householder QR, for the FP64-class precision modes.
//
// Same algorithm as the FP64 cluster panel in qr.cu (rows of the panel split over the CTAs of
// one thread-block cluster, one exchange of partial sums per column through distributed shared memory, LAPACK dgeqr2 reflectors and the forward/columnwise dlarft T
// factor), with every per-element operation in double-FP32 arithmetic on the FP32 pipe. On
// this part the FP64 pipe issues about 2 FMA per clock per SM against 128 for FP32, and in the
// FP64 kernel the per-column update of the remaining panel columns is bound by it.
//
// Numbers are (hi, lo) float pairs (relative error ~2^-47 per operation, the standard model
// with u ~ 2^-47, so the factorisation stays backward stable at that level). The layout and
// schedule are chosen for short dependency chains on the FP32 pipe:
//   * 16 warps, each with four panel columns, (hi, lo) pairs interleaved in shared memory;
//     dot products accumulate compensated (hi, lo) sums renormalised once at the end;
//   * the CL partial sums of a column are added as a fixed binary tree (every CTA derives
//     bitwise-identical column scalars);
//   * the column scalars use 1 / norm from an rsqrtf seed refined by Newton steps in
//     double-FP32 (tau = 1 + |alpha| / norm needs no division; scale = sign / (norm tau) one
//     refined reciprocal), not FP64 square root and division;
//   * the T factor is distributed: CTA q extends rows a = q (mod CL) of T, so no CTA carries
//     a serial triangular product on the critical path, and two columns behind.
// Columns are scaled by powers of two at load (largest entry of each panel column near 2^32)
// so that squares and products of small entries stay inside the FP32 exponent range; QR of
// A D with D a power-of-two diagonal has the same reflectors and R D, so R entries are
// rescaled on store and reflectors, tau and T are unaffected.
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "tc_ptx.cuh"

namespace tnx {
namespace qrdf {

namespace cg = cooperative_groups;
using tc::mbar_arrive;
using tc::mbar_expect_tx;
using tc::mbar_init;
using tc::mbar_wait;
using tc::smem_u32;

constexpr int DPT = 512;  // threads per CTA
constexpr int PUSH = 1;   // sums are stored to every rank, to be awaited at a counting barrier
constexpr int PAD = 2;    // the row stride has PAD_ROWS zero rows below the CTA's own
constexpr int PAD_ROWS = 64;

struct df2 {
  float h, l;
};

// Error-free transformations with explicit roundings (no contraction into FMA, no reassociation)
__device__ __forceinline__ df2 two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
__device__ __forceinline__ df2 fast_two_sum(float a, float b) {  // |a| >= |b| or a == 0
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ df2 add(df2 x, df2 y) {
  const df2 s = two_sum(x.h, y.h);
  return fast_two_sum(s.h, __fadd_rn(s.l, __fadd_rn(x.l, y.l)));
}
__device__ __forceinline__ df2 neg(df2 x) { return {-x.h, -x.l}; }
__device__ __forceinline__ df2 mul(df2 x, df2 y) {
  const float p = __fmul_rn(x.h, y.h);
  float e = fmaf(x.h, y.h, -p);
  e = fmaf(x.h, y.l, e);
  e = fmaf(x.l, y.h, e);
  return fast_two_sum(p, e);
}
// x - w v
__device__ __forceinline__ df2 fms(df2 x, df2 w, df2 v) {
  const float p = __fmul_rn(w.h, v.h);
  float pe = fmaf(w.h, v.h, -p);
  pe = fmaf(w.h, v.l, pe);
  pe = fmaf(w.l, v.h, pe);
  const df2 s = two_sum(x.h, -p);
  return fast_two_sum(s.h, __fadd_rn(s.l, __fsub_rn(x.l, pe)));
}
// c += a b with c.l left unnormalised (long sums; renormalise with two_sum(c.h, c.l))
__device__ __forceinline__ void acc(df2& c, df2 a, df2 b) {
  const float p = __fmul_rn(a.h, b.h);
  float pe = fmaf(a.h, b.h, -p);
  pe = fmaf(a.h, b.l, pe);
  pe = fmaf(a.l, b.h, pe);
  const df2 s = two_sum(c.h, p);
  c.h = s.h;
  c.l = __fadd_rn(c.l, __fadd_rn(s.l, pe));
}
__device__ __forceinline__ df2 norm(df2 c) { return two_sum(c.h, c.l); }
// 1 / sqrt(t), t > 0: rsqrtf seed y (error ~2^-22) and one third-order step y + y (e / 2 + 3 e^2 / 8) on the
// double-FP32 residual e = 1 - t y^2, accurate to ~2^-47 absolutely: the correction, ~2^-22 of y, is
// enough in FP32
__device__ __forceinline__ df2 rsqrt_df(df2 t) {
  const float y = rsqrtf(t.h), yy = __fmul_rn(y, y);
  const df2 e = fms({1.f, 0.f}, t, {yy, fmaf(y, y, -yy)});
  return fast_two_sum(y, __fmul_rn(__fmul_rn(y, e.h), fmaf(0.375f, e.h, 0.5f)));
}
// 1 / b: approximate FP32 reciprocal seed z and one third-order step z + z (e + e^2), e = 1 - b z
__device__ __forceinline__ df2 rcp_df(df2 b) {
  const float z = __fdividef(1.f, b.h);
  const df2 e = fms({1.f, 0.f}, b, {z, 0.f});
  return fast_two_sum(z, __fmul_rn(__fmul_rn(z, e.h), 1.f + e.h));
}
__device__ __forceinline__ df2 shfl_xor(df2 x, int o) {
  return {__shfl_xor_sync(0xffffffffu, x.h, o), __shfl_xor_sync(0xffffffffu, x.l, o)};
}

// double (exponent lowered by e: x 2^-e, exact) -> (hi, lo); Inf and NaN stay non-finite
// (split_df gives (+-inf, 0) / (NaN, 0)) so that they propagate through the factorisation
__device__ __forceinline__ df2 split_scaled(double x, int e) {
  long long b = __double_as_longlong(x);
  const int ef = int((b >> 52) & 0x7ff);
  if (ef == 2047) {
    df2 r;
    split_df(x, r.h, r.l);
    return r;
  }
  if (ef == 0) {  // zero / subnormal (below 2^-1022: far below the split's range)
    b &= (1LL << 63);
  } else if (ef - e <= 0) {
    b &= (1LL << 63);
  } else {
    b -= (long long)e << 52;
  }
  df2 r;
  split_df(__longlong_as_double(b), r.h, r.l);
  return r;
}
// (hi, lo) -> double x 2^e
__device__ __forceinline__ double join_scaled(df2 x, int e) {
  const double d = join_df(x.h, x.l);
  long long b = __double_as_longlong(d);
  const int ef = int((b >> 52) & 0x7ff);
  if (ef == 0 || e == 0) return d;
  const int ne = ef + e;
  if (ne >= 2047) return __longlong_as_double((b & (1LL << 63)) | (0x7ffLL << 52));
  if (ne <= 0) return __longlong_as_double(b & (1LL << 63));
  return __longlong_as_double(b + ((long long)e << 52));
}

__device__ __forceinline__ void cluster_arrive_release() {
  asm volatile("barrier.cluster.arrive.release;\n" ::: "memory");
}
__device__ __forceinline__ void cluster_wait_acquire() {
  asm volatile("barrier.cluster.wait.acquire;\n" ::: "memory");
}

// 8 bytes into the shared memory of `rank` at this CTA's address `at`, counted by that CTA's barrier `bar`
__device__ __forceinline__ void send_async(uint32_t at, df2 x, uint32_t bar, int rank) {
  asm volatile(
      "{\n .reg .b32 a, b;\n mapa.shared::cluster.u32 a, %0, %4;\n mapa.shared::cluster.u32 b, %3, %4;\n"
      " st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [a], {%1, %2}, [b];\n}\n" ::"r"(at),
      "f"(x.h), "f"(x.l), "r"(bar), "r"(rank)
      : "memory");
}

__device__ __forceinline__ void send_async(uint32_t at, double x, uint32_t bar, int rank) {
  asm volatile(
      "{\n .reg .b32 a, b;\n mapa.shared::cluster.u32 a, %0, %3;\n mapa.shared::cluster.u32 b, %2, %3;\n"
      " st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [a], %1, [b];\n}\n" ::"r"(at),
      "l"(__double_as_longlong(x)), "r"(bar), "r"(rank)
      : "memory");
}

// Dynamic shared memory bytes of one CTA: (hi, lo) pairs of the panel [NB][ld] (interleaved pairs: one
// 64-bit access per operand) and the exchange of two steps, sums [ranks][NB] and the pivot row [NB]: with `push` every rank's
// sums, without it this rank's, which the others read.
template <int NB, int CL>
constexpr size_t panel_df_smem_bytes(int ld, bool push) {
  return (size_t(NB) * size_t(ld) + 2 * size_t(NB) * ((push ? CL : 1) + 1)) * sizeof(df2);
}

// Factor panel columns [j0, j0+nb) of the column-major m x n matrix F (ld = m), rows >= j0:
// on exit R on/above the diagonal, the reflectors below it (unit diagonal implicit), tau, and T
// (column-major, ld NB, upper triangular; zero outside [0, nb)) with H_j0..H_{j0+nb-1} =
// I - V T V^T. `ld` is the CTA's shared-memory row stride (>= rows per CTA).
//
// What bounds a column: the chain exchange - scalars - reflector - update, of which the update's arithmetic
// is under a third. So
//   * a CTA stores its sums to every rank (PUSH), counted by a barrier in the receiver's shared memory: a
//     cluster barrier, whose release and acquire took 2400 cycles a column, is not needed, and the sums
//     are read at local latency. Panels too tall for that buffer read them from the ranks;
//   * warp 0 takes the two sums that the scalars need straight from the exchange while others fetch the rest;
//   * v and column jj+1 are formed in place; threads that stand for the columns meanwhile compute the
//     factors of the update and send the next pivot row; T follows two columns behind;
//   * in the update a warp has its columns whole: v and the next column are read once for four columns,
//     and no warp goes through the update, the norm and the T dots one after the other. Zero rows below
//     the CTA's own (PAD, where they fit) spare it the bounds checks, a third of its instructions.
// The 16 panels of a 2048 x 1024 matrix: 280 us each with five block barriers and a cluster barrier a
// column, 254 us so. 256 or 1024 threads: a quarter slower.
template <int NB, int CL, int MODE>
__global__ void __launch_bounds__(DPT) panel_df_kernel(double* __restrict__ F, int64_t m, int64_t j0, int nb, int ld,
                                                       double* __restrict__ tau_out, double* __restrict__ T_out) {
  constexpr int NW = DPT / 32, CPW = NB / NW;  // warp w works on columns w, w + NW, ...: CPW of them
  constexpr int GL = 32 / CPW;                 // lanes that end up with a column's sum
  constexpr int NR = NB / CL;                  // rows of T held by each CTA
  static_assert(NB % CL == 0 && NB <= 64 && CPW >= 1 && CPW * NW == NB && 2 * CL <= 32 && 4 + NR <= NW, "panel shape");
  cg::cluster_group cluster = cg::this_cluster();
  const int q = int(cluster.block_rank());
  extern __shared__ df2 pd[];
  df2* X = pd;                        // [NB][ld] panel rows of this CTA, column-major
  constexpr bool push = MODE & PUSH, pad = MODE & PAD;
  df2* part = pd + NB * ld;           // exchange [2][push ? CL : 1][NB]: dots (right of the column) and T dots (left)
  constexpr int pr = push ? CL : 1;
  df2* prow = part + 2 * pr * NB;     // [2][NB] pivot row (pushed, or the owner's)
  __shared__ unsigned long long smax[NB];
  __shared__ df2 W[NB], Z[2][NB], taus[NB], sc[4];  // W: factors of the current reflector in the columns right of it
  __shared__ df2 Tr[NR][NB];          // rows q, q + CL, ... of T
  __shared__ int cexp[NB];
  __shared__ __align__(8) uint64_t bars[2];  // arrival of a step's sums and end of the update before it (push)
  __shared__ int s_dead;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ci = warp + NW * (lane / GL), h = lane % GL;
  constexpr int CT = 64;  // threads CT .. CT + NB - 1 stand for the columns before and after the scalars
  const int64_t mp = m - j0;
  const int rpc = int((mp + CL - 1) / CL);
  const int r0 = q * rpc;
  const int rows = int(r0 >= mp ? 0 : (mp - r0 < rpc ? mp - r0 : rpc));

  // ---- column scales: largest |entry| of each panel column over the cluster (integer max of
  // the magnitude bits), exponent chosen so that it lands in [2^31, 2^32)
  {
    const uint32_t bar = smem_u32(bars);
    if (push && tid == 0) {
      s_dead = 0;
      mbar_init(bar, 1 + NW);
      mbar_init(bar + 8, 1 + NW);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      mbar_expect_tx(bar, uint32_t(8 * nb * (CL + 1)));
      mbar_expect_tx(bar + 8, uint32_t(8 * ((nb - 1) * CL + nb - 1)));
    }
    unsigned long long mx = 0;
    if (ci < nb)
      for (int r = h; r < rows; r += GL) {
        const unsigned long long b =
            static_cast<unsigned long long>(__double_as_longlong(F[(j0 + ci) * m + j0 + r0 + r])) & 0x7fffffffffffffffull;
        mx = b > mx ? b : mx;
      }
#pragma unroll
    for (int o = GL / 2; o > 0; o >>= 1) {
      const unsigned long long t = __shfl_xor_sync(0xffffffffu, mx, o);
      mx = t > mx ? t : mx;
    }
    if (h == 0 && ci < NB) smax[ci] = mx;
  }
  cluster_arrive_release();
  cluster_wait_acquire();
  if (tid < NB) {
    unsigned long long mx = 0;
#pragma unroll
    for (int r = 0; r < CL; ++r) {
      const unsigned long long t = cluster.map_shared_rank(smax, r)[tid];
      mx = t > mx ? t : mx;
    }
    const int ef = int(mx >> 52);  // biased exponent of the column maximum (0: zero column)
    cexp[tid] = ef == 0 ? 0 : ef - 1023 - 31;
  }
  __syncthreads();
  for (int e = tid; e < nb * rows; e += DPT) {
    const int c = e / rows, r = e % rows;
    X[c * ld + r] = split_scaled(F[(j0 + c) * m + j0 + r0 + r], cexp[c]);
  }
  if (pad)
    for (int e = tid; e < NB * PAD_ROWS; e += DPT) X[(e / PAD_ROWS) * ld + rows + e % PAD_ROWS] = {0.f, 0.f};
  for (int e = tid; e < NR * NB; e += DPT) Tr[e / NB][e % NB] = {0.f, 0.f};
  // column k of the rows of T held by warps 4 .. 4 + NR - 1: T[a][k] = -tau_k sum_{a <= c < k} T[a][c] z_c,
  // T[k][k] = tau_k
  auto extend_t = [&](int k) {
    const int row = warp - 4, a = q + CL * row;
    if (k < 0) return;
    if (a < k) {
      df2 t = {0.f, 0.f};
      for (int c = a + lane; c < k; c += 32) acc(t, Tr[row][c], Z[k & 1][c]);
      t = norm(t);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t = add(t, shfl_xor(t, o));
      if (lane == 0) Tr[row][k] = neg(mul(taus[k], t));
    } else if (a == k && lane == 0) {
      Tr[row][k] = taus[k];
    }
  };
  // a column's sum, held by the GL lanes of column ci, into the exchange
  auto send_sum = [&](int buf, df2 sum) {
    if (push) {
#pragma unroll
      for (int r = h; r < CL; r += GL)
        send_async(smem_u32(&part[(buf * CL + q) * NB + ci]), sum, smem_u32(&bars[buf]), r);
    } else if (h == 0) {
      part[buf * NB + ci] = sum;
    }
  };
  // column c's entry in the next pivot row
  auto send_pivot = [&](int buf, int c, df2 piv) {
    if (push) {
      const uint32_t at = smem_u32(&prow[buf * NB + c]), bar = smem_u32(&bars[buf]);
#pragma unroll 4
      for (int r = 0; r < CL; ++r) send_async(at, piv, bar, r);
    } else {
      prow[buf * NB + c] = piv;
    }
  };
  // A warp's end of the update that sends into buffer buf: its stores to the panel come before this CTA reads what the
  // barrier guards (the sums order the stores of the lane that sends them alone)
  auto updated = [&](int buf) {
    if (push) {
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bars[buf]));
    }
  };
  // before the exchange of step `step`, or the panel as the update before left it, is read
  auto await = [&](int step) {
    if (push && !mbar_wait(smem_u32(&bars[step & 1]), (step >> 1) & 1)) s_dead = 1;
  };
  auto exchange = [&] {
    if (!push) {
      cluster_arrive_release();
      cluster_wait_acquire();
    }
  };
  auto partial = [&](int buf, int r, int idx) {
    return push ? part[(buf * CL + r) * NB + idx] : cluster.map_shared_rank(part, r)[buf * NB + idx];
  };
  // sum of the CL partials idx as a fixed binary tree
  auto tree_sum = [&](int buf, int idx) {
    df2 v[CL];
#pragma unroll
    for (int r = 0; r < CL; ++r) v[r] = partial(buf, r, idx);
#pragma unroll
    for (int s = 1; s < CL; s <<= 1)
#pragma unroll
      for (int r = 0; r + s < CL; r += 2 * s) v[r] = add(v[r], v[r + s]);
    return v[0];
  };
  auto pivot = [&](int buf, int owner, int idx) {
    return push ? prow[buf * NB + idx] : cluster.map_shared_rank(prow, owner)[buf * NB + idx];
  };
  auto from_lane = [&](df2 x, int l) {
    return df2{__shfl_sync(0xffffffffu, x.h, l), __shfl_sync(0xffffffffu, x.l, l)};
  };
  // sums of the warp's columns over its lanes: the GL lanes of column ci get that of ci
  auto reduce = [&](df2* a) {
    int o = 16;
#pragma unroll
    for (int n = CPW; n > 1; n >>= 1, o >>= 1)
#pragma unroll
      for (int i = 0; i < n / 2; ++i) {
        const bool up = lane & o;
        const df2 give = up ? a[i] : a[i + n / 2], keep = up ? a[i + n / 2] : a[i];
        a[i] = add(keep, shfl_xor(give, o));
      }
#pragma unroll
    for (o = GL / 2; o > 0; o >>= 1) a[0] = add(a[0], shfl_xor(a[0], o));
    return a[0];
  };
  __syncthreads();
  // partials of pivot 0: x_0 . x_c below row 0, and pivot row 0 (rank 0)
  {
    df2 a[CPW];
#pragma unroll
    for (int k = 0; k < CPW; ++k) a[k] = {0.f, 0.f};
    for (int r = lane; r < rows; r += 32) {
      const df2 x0 = r0 + r > 0 ? X[r] : df2{0.f, 0.f};
#pragma unroll
      for (int k = 0; k < CPW; ++k)
        if (warp + NW * k < nb) acc(a[k], x0, X[(warp + NW * k) * ld + r]);
    }
#pragma unroll
    for (int k = 0; k < CPW; ++k) a[k] = norm(a[k]);
    const df2 sum = reduce(a);
    if (ci < nb) send_sum(0, sum);
    if (r0 == 0 && rows > 0 && tid < nb) send_pivot(0, tid, X[tid * ld]);
    updated(0);
  }
  exchange();

  for (int jj = 0; jj < nb; ++jj) {
    const int par = jj & 1;
    const int owner = jj / rpc;
    const bool has_next = jj + 1 < nb;
    const int lj = jj - r0, ln = lj + 1;  // local rows of pivots jj and jj + 1 (outside [0, rows) on other CTAs)
    const bool has_lj = lj >= 0 && lj < rows, has_ln = ln >= 0 && ln < rows;
    df2 sum_c = {0.f, 0.f}, piv_c = {0.f, 0.f}, xl_j = {0.f, 0.f}, xl_c = {0.f, 0.f};
    if (warp == 0) {
      await(jj);
      if (push && lane == 0 && jj + 2 <= nb)  // the buffer's next use, for step jj + 2
        mbar_expect_tx(smem_u32(&bars[par]), uint32_t(8 * ((nb - 1) * CL + nb - 2 - jj)));
      // ---- column scalars, from the sums of columns jj and jj + 1 (the halves of 2 CL lanes)
      const int c = jj + (((lane / CL) & 1) && has_next ? 1 : 0);
      df2 t = partial(par, lane % CL, c);
      const df2 alpha = pivot(par, owner, jj), pn = pivot(par, owner, has_next ? jj + 1 : jj);
#pragma unroll
      for (int o = 1; o < CL; o <<= 1) t = add(t, shfl_xor(t, o));
      const df2 sigma = from_lane(t, 0), sn = from_lane(t, CL);
      df2 tj = {0.f, 0.f}, beta = alpha, scale = {0.f, 0.f};
      if (sigma.h != 0.f || sigma.l != 0.f) {
        // nrm = sqrt(alpha^2 + sigma) through y = 1 / nrm: tau = (beta - alpha) / beta =
        // 1 + |alpha| y, scale = 1 / (alpha - beta) = sign(alpha) y / tau
        const df2 t2 = add(mul(alpha, alpha), sigma);
        const df2 y = rsqrt_df(t2);
        const df2 nrm = mul(t2, y);
        const bool pos = alpha.h > 0.f || (alpha.h == 0.f && alpha.l >= 0.f);
        beta = pos ? neg(nrm) : nrm;
        tj = add({1.f, 0.f}, mul(pos ? alpha : neg(alpha), y));
        const df2 sy = mul(y, rcp_df(tj));
        scale = pos ? sy : neg(sy);
      }
      const df2 wn = has_next ? mul(tj, add(pn, mul(scale, sn))) : df2{0.f, 0.f};
      if (lane == 0) {
        sc[0] = tj;
        sc[1] = beta;
        sc[2] = scale;
        sc[3] = wn;
        taus[jj] = tj;
      }
    } else if (tid >= CT && tid < CT + NB) {
      // ---- meanwhile: sum and pivot entry of column c >= jj + 2, T dots Z[a] = v_a . v_{jj-1} (a < jj - 1)
      const int c = tid - CT;
      await(jj);
      if (c > jj + 1 && c < nb) {
        sum_c = tree_sum(par, c);
        piv_c = pivot(par, owner, c);
      } else if (c < jj - 1) {
        Z[par ^ 1][c] = tree_sum(par, c);
      }
      if (has_ln && c < nb) {  // row jj + 1 before the update
        xl_j = X[jj * ld + ln];
        xl_c = X[c * ld + ln];
      }
    } else if (warp >= 4 && warp < 4 + NR) {
      extend_t(jj - 2);
    }
    __syncthreads();
    if (push && s_dead) break;
    const df2 tj = sc[0], scale = sc[2];
    const int rA = lj > 0 ? lj : 0;
    df2* xj = X + jj * ld;
    df2* xn = xj + ld;
    // ---- phase A: v = scale x_jj below the pivot (beta at it, where v is 1), next column updated by it
    {
      const df2 wn = sc[3], beta = sc[1];
      for (int r = rA + tid; r < rows; r += DPT) {
        const bool at = r == lj;
        const df2 v = at ? df2{1.f, 0.f} : mul(scale, xj[r]);
        if (has_next) xn[r] = fms(xn[r], wn, v);
        xj[r] = at ? beta : v;
      }
    }
    // meanwhile: the columns' factors, and the next pivot row on its way
    if (tid >= CT && tid < CT + NB) {
      const int c = tid - CT;
      if (c > jj && c < nb) {
        const df2 w = c == jj + 1 ? sc[3] : mul(tj, add(piv_c, mul(scale, sum_c)));
        W[c] = w;
        if (has_lj && c > jj + 1) X[c * ld + lj] = add(X[c * ld + lj], neg(w));  // v_jj[jj] = 1
        if (has_ln) {
          const df2 p = fms(xl_c, w, mul(scale, xl_j));
          if (c > jj + 1) X[c * ld + ln] = p;
          send_pivot(par ^ 1, c, p);
        }
      } else if (c < jj && (has_lj || has_ln)) {  // the pivots' rows of the T dots
        df2 z = {0.f, 0.f};
        if (has_lj) z = X[c * ld + lj];
        if (has_ln) acc(z, xl_c, mul(scale, xl_j));
        W[c] = norm(z);
      }
    }
    __syncthreads();
    // ---- phase B: update columns c > jj + 1 and the partial dots of step jj + 1 (norm of
    // column jj + 1 below its pivot, its dots with c > jj + 1), T dots. A lane has rows lane, lane + 32, ..
    // of all the warp's columns, two at a time, from the first row below both pivots on
    df2 a[CPW], wk[CPW];
#pragma unroll
    for (int k = 0; k < CPW; ++k) {
      a[k] = {0.f, 0.f};
      wk[k] = W[warp + NW * k];  // not used left of the update
    }
    auto two_rows = [&](int r, auto whole) {
      constexpr bool all = decltype(whole)::value;  // both rows exist (or are zero rows of the padding)
      const int r1 = r + 32;
      const bool i0 = all || r < rows, i1 = all || r1 < rows;
      const df2 zero = {0.f, 0.f};
      const df2 v0 = i0 ? xj[r] : zero, v1 = i1 ? xj[r1] : zero;
      const df2 d0 = i0 && has_next ? xn[r] : zero, d1 = i1 && has_next ? xn[r1] : zero;
#pragma unroll
      for (int k = 0; k < CPW; ++k) {
        const int c = warp + NW * k;
        df2* xc = X + c * ld;
        if (c >= nb || c == jj) continue;
        if (c == jj + 1) {
          acc(a[k], d0, d0);
          acc(a[k], d1, d1);
          continue;
        }
        const df2 x0 = i0 ? xc[r] : zero, x1 = i1 ? xc[r1] : zero;
        if (c > jj) {
          const df2 t0 = fms(x0, wk[k], v0), t1 = fms(x1, wk[k], v1);
          if (i0) xc[r] = t0;
          if (i1) xc[r1] = t1;
          acc(a[k], d0, t0);
          acc(a[k], d1, t1);
        } else {
          acc(a[k], x0, v0);
          acc(a[k], x1, v1);
        }
      }
    };
    for (int r = lj + 2 > 0 ? lj + 2 : 0; r < rows; r += 64) {
      if (pad || r + 64 <= rows) two_rows(r + lane, std::true_type{});
      else two_rows(r + lane, std::false_type{});
    }
#pragma unroll
    for (int k = 0; k < CPW; ++k) a[k] = norm(a[k]);
    df2 sum = reduce(a);
    if (ci < jj && (has_lj || has_ln)) sum = add(sum, W[ci]);
    if (ci < nb && ci != jj) send_sum(par ^ 1, sum);
    updated(par ^ 1);
    exchange();
  }
  // the last two columns of T, the last one from the final exchange
  __syncthreads();
  if (tid < NB) {
    if (!s_dead) await(nb);
    if (tid < nb - 1) Z[(nb - 1) & 1][tid] = tree_sum(nb & 1, tid);
  } else if (warp >= 4 && warp < 4 + NR) {
    extend_t(nb - 2);
  }
  __syncthreads();
  if (warp >= 4 && warp < 4 + NR) extend_t(nb - 1);
  __syncthreads();
  // T (column-major, ld NB): this CTA's rows; tau from rank 0
  for (int e = tid; e < NR * NB; e += DPT) {
    const int i = e / NB, b = e % NB, a = q + CL * i;
    T_out[b * NB + a] = (a <= b && b < nb) ? join_df(Tr[i][b].h, Tr[i][b].l) : 0.0;
  }
  const bool dead = push && s_dead;  // a bounded wait ran out: NaN, so that no caller takes the result
  if (q == 0)
    for (int b = tid; b < NB; b += DPT) tau_out[b] = b < nb ? join_df(taus[b].h, taus[b].l) : 0.0;
  const double nan = __longlong_as_double(0x7ff8000000000000LL);
  // panel back to F: R entries (panel row <= column) rescaled, reflectors as they are
  for (int e = tid; e < nb * rows; e += DPT) {
    const int c = e / rows, r = e % rows;
    const df2 v = X[c * ld + r];
    F[(j0 + c) * m + j0 + r0 + r] = dead ? nan : (r0 + r <= c ? join_scaled(v, cexp[c]) : join_df(v.h, v.l));
  }
  if (dead) __nanosleep(1000000);  // stores of this CTA may still be on their way to others
  // no CTA leaves while another may still read its slots
  cluster_arrive_release();
  cluster_wait_acquire();
}

}  // namespace qrdf
}  // namespace tnx
