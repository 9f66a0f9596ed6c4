// FP64-class GEMM on the tcgen05 tensor cores by exact integer slicing (Ozaki scheme).
//
//   C = alpha op(A) op(B) + beta C,   FP64 in and out.
//
// Row i of op(A) is scaled by 2^-ea_i so that its entries are below 1/2 in magnitude and cut, by
// integer extraction from the 53-bit mantissa in signed fixed point, into S = 8 balanced base-128
// digits (each rounded to nearest, so the remainder after digit s is at most half a unit of it):
//   op(A)_ik 2^-ea_i = sum_{s<S} qa_s,ik 2^-7(s+1) + r_ik,   |r_ik| <= 2^-57,   |qa_s,ik| <= 64,
// integers that BF16 holds exactly. Column j of op(B) likewise with eb_j. Then
//   C_ij = 2^(ea_i + eb_j) sum_{g<S} 2^-7(g+2) P_g,ij + O(2^-53) per product,
//   P_g,ij = sum_{s+t=g} sum_k qa_s,ik qb_t,kj                          (36 slice pairs),
// and every P_g is a sum of integer products of magnitude at most 2^12. Over KC = 480 values of
// k the partial sum of a group (at most 8 pairs) stays below 8 * 480 * 2^12 < 2^24, so the FP32
// accumulation of the tensor cores in tensor memory is exact; every KC the eight group
// accumulators are drained into a double-FP32 running sum per output (epilogue warps), scaled
// by 2^-7(g+2). (Unbalanced 7-bit digits up to 127 would allow only KC = 128: the drains, which
// stall the MMAs, are 3.75x rarer with balanced ones.)
// Error: ~2^-52 per product relative to 2^ea_i 2^eb_j (the row / column maxima), plus the
// double-FP32 summation (~2^-46 of the running sum): FP64-class where rows and columns do not
// span many decades; at the tensor cores' rate divided by 36.
//
// Kernel: 128 x 64 output tiles, 10 warps: warp 0 TMA producer (all 2 S slice tiles of
// a 32-deep K block per stage, 2 stages of 96 KB, 64-byte swizzle), warp 1 TMEM allocation (512
// columns: eight 64-column group accumulators) and tcgen05.mma issue of the 36
// slice products per K block as 12 MMAs per 16-deep step (slice q of A against the B slices
// 0..7-q at once, N up to 256), warps 2-9 epilogue (two per TMEM lane quarter, 32 columns
// each). All
// mbarrier waits are bounded (~2 s); on expiry the kernel raises the error flag and returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "tc_ptx.cuh"
#include "tnx_internal.cuh"

namespace tnx {
namespace {

using namespace tc;

constexpr int OZ_S = 8;                         // slices per operand
constexpr int OZ_BM = 128, OZ_BN = 64, OZ_BK = 32;  // BK = 32 bf16 = one 64-byte swizzle row
constexpr int OZ_KC = 480;                      // K values per exact accumulation chunk
constexpr int OZ_STAGES = 2;                    // a stage holds all 2 S slice tiles of one K block
constexpr int OZ_PARTS = 3;                      // parts in which a stage is freed
constexpr int OZ_EPI_WARPS = 8;                 // two per TMEM lane quarter, 32 columns each
constexpr int OZ_THREADS = 64 + 32 * OZ_EPI_WARPS;
constexpr uint32_t OZ_TMEM_COLS = 512;

// ---------------------------------------------------------------- operand slicing
// Logical operand X(r, k) = src[r * rs + k * ks], rows x K (FP64). bmax[r] (zeroed before) =
// largest biased FP64 exponent in row r, by atomicMax over CTAs of 32 rows x OZ_SCAN_K values of
// k (the scan runs over the whole grid, not one CTA per row block). The row's scale exponent is
// E = bmax - 1021 (|X(r, k)| < 2^(E-1)), 0 for an all-zero row: row_scale_exp. bmax = 2047 marks
// a row with Inf or NaN, whose outputs the GEMM epilogue sets to NaN.
constexpr int OZ_SCAN_K = 256;
__device__ __forceinline__ int exp_field(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }

// KC: k is the unit-stride index of src (a warp per row, lanes along k), otherwise r is (lanes along r,
// a warp per k). 32 rows x OZ_SCAN_K values a CTA, eight loads in flight a thread.
template <bool KC>
__global__ void __launch_bounds__(256) oz_rowmax_kernel(const double* __restrict__ src, int64_t rows, int64_t K,
                                                        int64_t rs, int64_t ks, int* __restrict__ bmax, int64_t s_src,
                                                        int64_t s_bmax, const int* __restrict__ mask) {
  __shared__ int part[8][32];
  if (mask && !mask[blockIdx.z]) return;  // a chain the caller masked out
  src += int64_t(blockIdx.z) * s_src;
  bmax += int64_t(blockIdx.z) * s_bmax;
  const int64_t r0 = int64_t(blockIdx.y) * 32, kb = int64_t(blockIdx.x) * OZ_SCAN_K;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (KC) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int64_t r = r0 + warp * 4 + i;
      int best = 0;  // biased exponent, 0 = zero / denormal
      if (r < rows) {
        double x[OZ_SCAN_K / 32];
#pragma unroll
        for (int j = 0; j < OZ_SCAN_K / 32; ++j) {
          const int64_t k = kb + j * 32 + lane;
          x[j] = k < K ? src[r * rs + k] : 0.0;
        }
#pragma unroll
        for (int j = 0; j < OZ_SCAN_K / 32; ++j) best = max(best, exp_field(x[j]));
      }
      best = __reduce_max_sync(0xffffffffu, best);
      if (lane == 0 && best > 0) atomicMax(&bmax[r], best);
    }
  } else {
    const int64_t r = r0 + lane;
    int best = 0;
    if (r < rows) {
      for (int j0 = 0; j0 < OZ_SCAN_K / 8; j0 += 8) {
        double x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int64_t k = kb + (j0 + j) * 8 + warp;
          x[j] = k < K ? src[r + k * ks] : 0.0;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) best = max(best, exp_field(x[j]));
      }
    }
    part[warp][lane] = best;
    __syncthreads();
    if (warp == 0 && r < rows) {
#pragma unroll
      for (int i = 1; i < 8; ++i) best = max(best, part[i][lane]);
      if (best > 0) atomicMax(&bmax[r], best);
    }
  }
}

__device__ __forceinline__ int row_scale_exp(int bmax) { return bmax > 0 ? bmax - 1021 : 0; }

// planes[s][r][k] (row pitch Kp, rows_pad rows per plane) = slice s of X(r, k) 2^-E[r];
// zero for r >= rows or k >= K.
//
// The slices are written once and read by TMA, 16 bytes an element against the 8 read, so this is
// bound by memory as long as an element costs few instructions: with x 2^-E as X in signed fixed point
// (63 fraction bits, |X| < 2^62), the balanced digits q_0 .. q_7 of X = sum q_s 2^(56 - 7s) + remainder
// are those of Y = X + sum_s 2^(55 - 7s) in plain base 128, less 64 each (the first one as it
// is): one 64-bit addition instead of a rounded shift and a subtraction per digit. A digit becomes a float by
// OR-ing it into the mantissa of 1.5 2^23 and subtracting that, and its upper half is the BF16 value.
// A thread converts two neighbouring k of a row and stores them as one word. 19.9 M elements of a
// chi = 1024 environment update: 217 us with a digit's rounding, sign and exponent formed apart
// and 2-byte stores, 91 us so (71 us the bytes at the copy's rate); the row maxima 41 us, 97 us by
// one warp of each CTA from a staged tile.
template <bool KC>
__global__ void __launch_bounds__(256) oz_slice_kernel(const double* __restrict__ src, int64_t rows, int64_t K,
                                                       int64_t rs, int64_t ks, const int* __restrict__ exps,
                                                       uint16_t* __restrict__ planes, int64_t rows_pad, int64_t Kp,
                                                       int64_t s_src, const int* __restrict__ mask) {
  __shared__ double tile[32][65];  // [r][k], 32 rows x 64 values of k
  if (mask && !mask[blockIdx.z]) return;
  src += int64_t(blockIdx.z) * s_src;
  exps += int64_t(blockIdx.z) * rows_pad;
  planes += int64_t(blockIdx.z) * OZ_S * rows_pad * Kp;
  const int64_t r0 = int64_t(blockIdx.y) * 32, k0 = int64_t(blockIdx.x) * 64;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double x[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int64_t r = KC ? r0 + warp * 4 + (i >> 1) : r0 + lane, k = KC ? k0 + (i & 1) * 32 + lane : k0 + i * 8 + warp;
    x[i] = (r < rows && k < K) ? (KC ? src[r * rs + k] : src[r + k * ks]) : 0.0;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (KC) tile[warp * 4 + (i >> 1)][(i & 1) * 32 + lane] = x[i];
    else tile[lane][i * 8 + warp] = x[i];
  }
  __syncthreads();
  const int64_t k = k0 + 2 * lane;
  if (k >= Kp) return;  // Kp is even
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int lr = warp * 4 + i;
    const int64_t r = r0 + lr;  // < rows_pad, a multiple of 32
    const int E = row_scale_exp(exps[r]);
    unsigned long long Y[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const unsigned long long u = static_cast<unsigned long long>(__double_as_longlong(tile[lr][2 * lane + h]));
      const int eb = int(u >> 52) & 0x7ff;
      const unsigned long long m53 = (u & ((1ull << 52) - 1)) | (1ull << 52);
      const int shift = eb - 1012 - E;  // <= 9 since |x| < 2^(E-1)
      unsigned long long F = shift >= 0 ? (m53 << (shift & 63)) : (shift > -64 ? (m53 >> -shift) : 0ull);
      if (eb == 0) F = 0ull;
      const unsigned long long X = (u >> 63) ? 0ull - F : F;
      Y[h] = X + 0x0081020408102040ull;  // sum over s of 2^(55 - 7s)
    }
    uint32_t* out = reinterpret_cast<uint32_t*>(planes + r * Kp + k);
#pragma unroll
    for (int s = 0; s < OZ_S; ++s) {
      const int sh = 56 - 7 * s;
      uint32_t w[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float f;
        if (s == 0) {  // signed top digit: -64 .. 64, kept in place by the bias of 128
          const uint32_t d = uint32_t(static_cast<long long>(Y[h]) >> sh) + 128u;
          f = __uint_as_float(0x4B400000u | d) - (12582912.f + 128.f);
        } else {
          const uint32_t d = uint32_t(Y[h] >> sh) & 127u;
          f = __uint_as_float(0x4B400000u | d) - (12582912.f + 64.f);
        }
        w[h] = __float_as_uint(f);
      }
      out[size_t(s) * rows_pad * Kp / 2] = __byte_perm(w[0], w[1], 0x7632);  // upper halves
    }
  }
}

// ---------------------------------------------------------------- GEMM kernel
// Stage layout (one K block of 32): A slices 0..S-1 (128 x 32 bf16, 8 KB each), then B slices
// 0..S-1 (64 x 32 bf16, 4 KB each), 64-byte swizzle; every slice tile is loaded once per K
// block and feeds all S(S+1)/2 slice products that use it. The B slice tiles lie back to back
// with the same 8-row swizzle groups, so B slices t0..t0+w-1 read as one (64 w) x 32 operand; the
// group accumulators lie back to back in TMEM (group g at column 64 g), so the products of A
// slice q with B slices t0..t0+w-1 land in groups q+t0..q+t0+w-1 by one MMA of N = 64 w. Per
// 16-deep step: A slice q against B slices 0..7-q in MMAs of N <= 256 (2, 2, 2, 2, 1, 1, 1, 1 for
// q = 0..7), 12 MMAs instead of 36, each A slice read from shared memory once or twice instead of
// 8 - q times.
// Batch and split-K: a work item is a tile of plane z = bz * nsplit + sz. Chain bz reads its slice planes at plane
// rows (bz * S + q) * Mp (A) / (bz * S + q) * Np (B) and its exponents at ea + bz Mp / eb + bz Np;
// split sz covers K blocks [sz kbs, (sz + 1) kbs). With nsplit == 1 the CTA writes
// C + bz sC = alpha P + beta C; otherwise the unscaled partial P to part[(sz * batch + bz) M N]
// (row-major, ld N), which oz_split_reduce_kernel sums in split order.
//
// One CTA an SM takes items until there are none: the producer draws them from a counter (a fixed share
// would leave the work of SMs that a concurrent kernel holds to the end) and hands them on through a
// queue of two. So the ring fills for the next tile, and its products run, while the epilogue warps
// are still at the FP64 sums and stores of this one; only the drain of the accumulators, which take all of
// tensor memory, stops the products (a tenth of the time at K = 1024). The whole MMA warp runs the issue loop, with
// descriptors in uniform registers. The products go by slices of A, so that a stage is freed in three parts
// (A slices 0-1, 2-3, 4-7 with the B slices that no later one meets) and the next block's copies start while it is
// still in use: 96 KB at about 64 bytes a clock and their latency take longer than the 2304 clocks of a block's
// products. 5120 x 2048 x 1024: 567 us with a launch of one CTA a tile and a one-lane issue loop, 485 us
// persistent, 458 us with stages freed in parts.
__global__ void __launch_bounds__(OZ_THREADS, 1)
    oz_gemm_kernel(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb, int M, int N,
                   int Kp, int Mp, int Np, const int* __restrict__ ea, const int* __restrict__ eb, double alpha,
                   double beta, double* __restrict__ C, int64_t ldc, int* __restrict__ err_flag,
                   int* __restrict__ counter, int batch, int nsplit, int kbs, int64_t sC, double* __restrict__ part,
                   const int* __restrict__ mask) {
  constexpr uint32_t A_TILE = OZ_BM * OZ_BK * 2, B_TILE = OZ_BN * OZ_BK * 2;
  constexpr uint32_t STAGE_BYTES = OZ_S * (A_TILE + B_TILE);
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full_bar[OZ_STAGES], empty_bar[OZ_STAGES][OZ_PARTS], chunk_full, chunk_empty, q_full[2], q_empty[2];
  __shared__ uint32_t tmem_base_sh;
  __shared__ int abort_sh, queue[2];
  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int tiles_n = Np / OZ_BN, tiles = tiles_n * (Mp / OZ_BM), items = tiles * batch * nsplit;
  const int kb_all = Kp / OZ_BK;
  const int kb_per_chunk = OZ_KC / OZ_BK;
  struct Item {
    int bz, sz, m0, n0, kb0, kblocks;
  };
  auto item = [&](int t) {
    Item w;
    const int z = t / tiles, r = t - z * tiles;
    w.bz = z / nsplit;
    w.sz = z - w.bz * nsplit;
    w.m0 = r / tiles_n * OZ_BM;
    w.n0 = r % tiles_n * OZ_BN;
    w.kb0 = w.sz * kbs;
    const int kb1 = min(kb_all, w.kb0 + kbs);
    w.kblocks = kb1 > w.kb0 ? kb1 - w.kb0 : 0;
    return w;
  };
  // w-th item of this CTA for a warp that consumes the queue; -1: no more (or a wait that ran out)
  auto next_item = [&](int w) {
    if (!mbar_wait(smem_u32(&q_full[w & 1]), (w >> 1) & 1)) {
      if (lane == 0) atomicExch(err_flag, 1);
      abort_sh = 1;
      return -1;
    }
    const int t = __shfl_sync(0xffffffffu, queue[w & 1], 0);
    if (lane == 0) mbar_arrive(smem_u32(&q_empty[w & 1]));
    return t;
  };

  if (threadIdx.x == 0) {
    for (int st = 0; st < OZ_STAGES; ++st) {
      mbar_init(smem_u32(&full_bar[st]), 1);
      for (int i = 0; i < OZ_PARTS; ++i) mbar_init(smem_u32(&empty_bar[st][i]), 1);
    }
    mbar_init(smem_u32(&chunk_full), 1);
    mbar_init(smem_u32(&chunk_empty), OZ_EPI_WARPS);
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&q_full[i]), 1);
      mbar_init(smem_u32(&q_empty[i]), 1 + OZ_EPI_WARPS);
    }
    abort_sh = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)),
                 "r"(OZ_TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base_sh, 0);

  if (warp == 0) {
    // ------------------------------------------------ TMA producer: one K block per stage
    if (lane == 0) {
      int issued = 0, t = blockIdx.x;
      bool ok = true;
      for (int w = 0; ok; ++w) {
        while (t < items && mask && !mask[t / tiles / nsplit]) t = int(gridDim.x) + atomicAdd(counter, 1);
        if (w >= 2 && !mbar_wait(smem_u32(&q_empty[w & 1]), ((w >> 1) & 1) ^ 1)) {
          atomicExch(err_flag, 1);
          abort_sh = 1;
          break;
        }
        queue[w & 1] = t < items ? t : -1;
        mbar_arrive(smem_u32(&q_full[w & 1]));
        if (t >= items) break;
        const Item it = item(t);
        t = int(gridDim.x) + atomicAdd(counter, 1);
        const int a_row = it.bz * OZ_S * Mp + it.m0, b_row = it.bz * OZ_S * Np + it.n0;
        for (int kb = 0; kb < it.kblocks; ++kb) {
          const int st = issued % OZ_STAGES;
          const uint32_t ph = (issued / OZ_STAGES) & 1;
          const uint32_t sa = base + st * STAGE_BYTES, sb = sa + OZ_S * A_TILE;
          const uint32_t fb = smem_u32(&full_bar[st]);
#pragma unroll
          for (int i = 0; i < OZ_PARTS; ++i) {
            if (ok && issued >= OZ_STAGES && !mbar_wait(smem_u32(&empty_bar[st][i]), ph ^ 1)) {
              atomicExch(err_flag, 1);
              abort_sh = 1;
            }
            ok = ok && !*((volatile int*)&abort_sh);
            if (!ok) break;
            if (i == 0) mbar_expect_tx(fb, STAGE_BYTES);
            // A slices q0 .. q1 - 1 and the B slices that no later one meets
            const int q0 = 2 * i, q1 = i == 2 ? OZ_S : 2 * i + 2;
#pragma unroll
            for (int q = q0; q < q1; ++q) {
              tma_load_2d(sa + q * A_TILE, &ta, fb, (it.kb0 + kb) * OZ_BK, a_row + q * Mp);
              const int t = OZ_S - 1 - q;
              tma_load_2d(sb + t * B_TILE, &tb, fb, (it.kb0 + kb) * OZ_BK, b_row + t * Np);
            }
          }
          ++issued;  // also a block given up half way: its wait below runs out long after its copies have landed
          if (!ok) break;
        }
      }
      for (int kb = issued - OZ_STAGES < 0 ? 0 : issued - OZ_STAGES; kb < issued; ++kb)
        mbar_wait(smem_u32(&full_bar[kb % OZ_STAGES]), (kb / OZ_STAGES) & 1);
    }
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer
    const uint64_t desc0 = smem_desc_sw64(base);
    const uint32_t full0 = smem_u32(full_bar), empty0 = smem_u32(empty_bar);
    const bool one = elect_one();
    int block = 0, chunk = 0;  // K blocks and chunks of all items so far
    bool ok = true;
    for (int w = 0; ok; ++w) {
      const int t = next_item(w);
      if (t < 0) break;
      const int kblocks = item(t).kblocks;
      for (int kb = 0; kb < kblocks && ok; ++chunk) {
        // the epilogue must have read the previous chunk's accumulators
        if (chunk > 0 && !mbar_wait(smem_u32(&chunk_empty), (chunk - 1) & 1)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        const int kb_end = min(kblocks, kb + kb_per_chunk);
        for (bool chunk_start = true; kb < kb_end; ++kb, ++block, chunk_start = false) {
          const int st = block % OZ_STAGES;
          if (!mbar_wait(full0 + 8 * st, (block / OZ_STAGES) & 1)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;");
          // addresses sit in the descriptors in units of 16 bytes
          const uint64_t da = desc0 + uint32_t(st) * (STAGE_BYTES >> 4), db = da + (OZ_S * A_TILE >> 4);
          if (one) {
#pragma unroll
            for (int q = 0; q < OZ_S; ++q) {
#pragma unroll
              for (int kk = 0; kk < OZ_BK / 16; ++kk) {
                const uint64_t ad = da + q * (A_TILE >> 4) + 2 * kk;
#pragma unroll
                for (int t0 = 0; t0 < OZ_S - q; t0 += 4) {
                  // slice pairs (q, t0) .. (q, t0 + w - 1) into groups q + t0 .. q + t0 + w - 1; the two
                  // MMAs of (q = 0, kk = 0) cover all eight groups and start a chunk's sums
                  const int w = OZ_S - q - t0 < 4 ? OZ_S - q - t0 : 4;
                  mma_bf16(tmem + uint32_t((q + t0) * OZ_BN), ad, db + t0 * (B_TILE >> 4) + 2 * kk,
                           instr_desc_bf16(OZ_BM, OZ_BN * w), (chunk_start && kk == 0 && q == 0) ? 0u : 1u);
                }
              }
              if (q == 1 || q == 3 || q == OZ_S - 1)
                mma_commit(empty0 + 8 * (st * OZ_PARTS + (q == 1 ? 0 : q == 3 ? 1 : 2)));
            }
          }
        }
        if (ok && one) mma_commit(smem_u32(&chunk_full));
      }
    }
    if (!ok) {
      if (one) atomicExch(err_flag, 1);
      abort_sh = 1;
    }
  } else {
    // ------------------------------------------------ epilogue (warps 2..9): tile row = lane of
    // the warp's TMEM lane quarter (warp mod 4), columns cb..cb+31 of every group (two warps a
    // quarter)
    const int quad = warp & 3;
    const int cb = (warp - 2) / 4 * 32;
    // a finished tile goes out through shared memory of the warp's own, 8 columns at a time, so that the
    // global stores are row segments: a thread holds one row of 32 columns
    constexpr int OW = 8, OLD = OW + 1;
    double* Cs = reinterpret_cast<double*>(smem_raw + (base - smem_u32(smem_raw)) + OZ_STAGES * STAGE_BYTES) +
                 (warp - 2) * 32 * OLD;
    const bool unit = alpha == 1.0;
    int chunk = 0;
    bool ok = true;
    for (int w = 0; ok; ++w) {
      const int t = next_item(w);
      if (t < 0) break;
      const Item it = item(t);
      const int nchunks = (it.kblocks + kb_per_chunk - 1) / kb_per_chunk;
      float hi[32], lo[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) hi[j] = lo[j] = 0.f;
      for (int c = 0; c < nchunks; ++c, ++chunk) {
        if (!mbar_wait(smem_u32(&chunk_full), chunk & 1)) {
          if (lane == 0) atomicExch(err_flag, 1);
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll 1
        for (int g = 0; g < OZ_S; g += 2) {  // two groups' loads in flight per wait
          uint32_t r[2][32];
          tmem_ld32_async(tmem + (uint32_t(quad * 32) << 16) + uint32_t(g * OZ_BN + cb), r[0]);
          tmem_ld32_async(tmem + (uint32_t(quad * 32) << 16) + uint32_t((g + 1) * OZ_BN + cb), r[1]);
          tmem_ld_wait();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float scale = __uint_as_float(uint32_t(127 - 7 * (g + h + 2)) << 23);  // 2^-7(g+h+2)
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const float v = __uint_as_float(r[h][j]) * scale;  // exact: power-of-two scaling
              float sum, err;
              two_sum_f(hi[j], v, sum, err);
              hi[j] = sum;
              lo[j] += err;
            }
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&chunk_empty));
      }
      if (!ok) break;
      // ea and eb are padded to Mp and Np entries
      const int row = it.m0 + quad * 32 + lane, col0 = it.n0 + cb;
      const int ear = ea[int64_t(it.bz) * Mp + row];
      const int* ebc = eb + int64_t(it.bz) * Np + col0;
      const int er = row_scale_exp(ear);
      const bool row_nonfinite = ear == 2047;  // the row holds Inf / NaN: its slices are not the value
      double* out = nsplit == 1 ? C + int64_t(it.bz) * sC : part + (int64_t(it.sz) * batch + it.bz) * M * N;
      const int64_t ldo = nsplit == 1 ? ldc : N;
      const int r0 = it.m0 + quad * 32 + (lane >> 3), cc = lane & 7;
#pragma unroll
      for (int p = 0; p < 32 / OW; ++p) {
#pragma unroll
        for (int j = 0; j < OW; ++j) {
          const int e = ebc[p * OW + j];
          // one FP64 addition an output; conversions and the power of two by integer arithmetic
          double v = scale_pow2(float_to_double(hi[p * OW + j]) + float_to_double(lo[p * OW + j]), er + row_scale_exp(e));
          if (row_nonfinite || e == 2047) v = __longlong_as_double(0x7ff8000000000000LL);
          Cs[lane * OLD + j] = v;
        }
        __syncwarp();
        const int c = col0 + p * OW + cc;
        if (c < N)
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int r = r0 + 4 * i;
            if (r < M) {
              double v = Cs[((lane >> 3) + 4 * i) * OLD + cc];
              double* o = out + int64_t(r) * ldo + c;
              if (nsplit == 1) {
                if (!unit) v *= alpha;
                if (beta != 0.0) v = fma(beta, *o, v);
              }
              *o = v;
            }
          }
        __syncwarp();
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(OZ_TMEM_COLS));
  }
}

// C[bz] = alpha sum_s part[s][bz] + beta C[bz] (split order fixed: deterministic)
__global__ void oz_split_reduce_kernel(const double* __restrict__ part, int nsplit, int batch, int M, int N,
                                       double alpha, double beta, double* __restrict__ C, int64_t ldc, int64_t sC,
                                       const int* __restrict__ mask) {
  const int bz = blockIdx.y;
  if (mask && !mask[bz]) return;
  const int64_t MN = int64_t(M) * N;
  for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < MN; e += int64_t(gridDim.x) * blockDim.x) {
    double v = 0.0;
    for (int s = 0; s < nsplit; ++s) v += part[(int64_t(s) * batch + bz) * MN + e];
    double* o = C + int64_t(bz) * sC + (e / N) * ldc + (e % N);
    v *= alpha;
    if (beta != 0.0) v = fma(beta, *o, v);
    *o = v;
  }
}

struct OzLayout {
  int64_t Mp, Np, Kp;
  uint16_t *sa, *sb;
  int *ea, *eb, *flag;
  double* part;
};

size_t oz_layout(int64_t m, int64_t n, int64_t k, int64_t batch, int nsplit, void* base, OzLayout* L) {
  OzLayout o;
  o.Mp = (m + OZ_BM - 1) / OZ_BM * OZ_BM;
  o.Np = (n + OZ_BN - 1) / OZ_BN * OZ_BN;
  o.Kp = (k + OZ_BK - 1) / OZ_BK * OZ_BK;
  size_t off = 0;
  auto take = [&](size_t bytes) { size_t r = off; off += align_up(bytes); return r; };
  const size_t osa = take(size_t(batch) * OZ_S * o.Mp * o.Kp * 2), osb = take(size_t(batch) * OZ_S * o.Np * o.Kp * 2),
               oea = take(size_t(batch) * o.Mp * 4), oeb = take(size_t(batch) * o.Np * 4), ofl = take(8),
               opt = take(nsplit > 1 ? size_t(nsplit) * batch * m * n * 8 : 0);
  if (base && L) {
    char* b = static_cast<char*>(base);
    o.sa = reinterpret_cast<uint16_t*>(b + osa);
    o.sb = reinterpret_cast<uint16_t*>(b + osb);
    o.ea = reinterpret_cast<int*>(b + oea);
    o.eb = reinterpret_cast<int*>(b + oeb);
    o.flag = reinterpret_cast<int*>(b + ofl);
    o.part = reinterpret_cast<double*>(b + opt);
    *L = o;
  }
  return off;
}

// stage ring, the epilogue warps' 32 x 9 doubles each, and slack for the alignment
size_t oz_smem_bytes() {
  return size_t(OZ_STAGES) * OZ_S * (OZ_BM * OZ_BK * 2 + OZ_BN * OZ_BK * 2) + OZ_EPI_WARPS * 32 * 9 * 8 + 1024;
}

}  // namespace

size_t gemm_oz_workspace_bytes(int64_t m, int64_t n, int64_t k) { return oz_layout(m, n, k, 1, 1, nullptr, nullptr); }
size_t gemm_oz_ex_workspace_bytes(int64_t m, int64_t n, int64_t k, int batch, int nsplit) {
  return oz_layout(m, n, k, batch, nsplit, nullptr, nullptr);
}

int gemm_oz_ex(bool ta, bool tb, int64_t m, int64_t n, int64_t k, double alpha, const double* A, int64_t lda,
               int64_t sA, const double* B, int64_t ldb, int64_t sB, double beta, double* C, int64_t ldc, int64_t sC,
               int batch, int nsplit, const int* mask, void* ws, size_t ws_bytes, cudaStream_t st) {
  if (m <= 0 || n <= 0 || batch <= 0) return TNX_OK;
  TNX_CHECK_ARG(nsplit >= 1 && batch <= 65535 && int64_t(batch) * nsplit <= 65535, "gemm_oz: batch %d x split %d",
                batch, nsplit);
  if (k <= 0) {
    if (batch == 1 && !mask) return gemm_f64(ta, tb, m, n, k, alpha, A, lda, 0, B, ldb, 0, beta, C, ldc, 0, 1, st);
    return gemm_f64(ta, tb, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch, st, 0, mask);
  }
  TNX_CHECK_SHAPE(int64_t(batch) * OZ_S * ((m + OZ_BM - 1) / OZ_BM * OZ_BM) < (int64_t(1) << 31) &&
                      int64_t(batch) * OZ_S * ((n + OZ_BN - 1) / OZ_BN * OZ_BN) < (int64_t(1) << 31),
                  "gemm_oz: operand too large");
  OzLayout L;
  const size_t need = oz_layout(m, n, k, batch, nsplit, ws, &L);
  if (!ws || ws_bytes < need) {
    set_error("gemm_oz: workspace %zu bytes < required %zu", ws_bytes, need);
    return TNX_ERR_WORKSPACE;
  }
  // op(A)(i, kk): ta ? A[kk lda + i] : A[i lda + kk];  op(B) column j: tb ? B[j ldb + kk] : B[kk ldb + j]
  const int64_t a_rs = ta ? 1 : lda, a_ks = ta ? lda : 1;
  const int64_t b_rs = tb ? ldb : 1, b_ks = tb ? 1 : ldb;
  // row maxima (atomicMax into zeroed arrays), the error flag and the item counter: ea, eb and flag are consecutive
  TNX_CUDA(cudaMemsetAsync(L.ea, 0, reinterpret_cast<char*>(L.flag + 2) - reinterpret_cast<char*>(L.ea), st));
  const unsigned kscan = unsigned((k + OZ_SCAN_K - 1) / OZ_SCAN_K), bzs = unsigned(batch);
  auto rowmax = [&](const double* src, int64_t rows, int64_t rs, int64_t ks, int* e, int64_t s_src, int64_t pad) {
    const dim3 grid(kscan, unsigned(pad / 32), bzs);
    if (ks == 1) oz_rowmax_kernel<true><<<grid, 256, 0, st>>>(src, rows, k, rs, ks, e, s_src, pad, mask);
    else oz_rowmax_kernel<false><<<grid, 256, 0, st>>>(src, rows, k, rs, ks, e, s_src, pad, mask);
  };
  auto slice = [&](const double* src, int64_t rows, int64_t rs, int64_t ks, const int* e, uint16_t* planes,
                   int64_t s_src, int64_t pad) {
    const dim3 grid(unsigned((L.Kp + 63) / 64), unsigned(pad / 32), bzs);
    if (ks == 1) oz_slice_kernel<true><<<grid, 256, 0, st>>>(src, rows, k, rs, ks, e, planes, pad, L.Kp, s_src, mask);
    else oz_slice_kernel<false><<<grid, 256, 0, st>>>(src, rows, k, rs, ks, e, planes, pad, L.Kp, s_src, mask);
  };
  rowmax(A, m, a_rs, a_ks, L.ea, sA, L.Mp);
  TNX_LAUNCH_CHECK();
  rowmax(B, n, b_rs, b_ks, L.eb, sB, L.Np);
  TNX_LAUNCH_CHECK();
  slice(A, m, a_rs, a_ks, L.ea, L.sa, sA, L.Mp);
  TNX_LAUNCH_CHECK();
  slice(B, n, b_rs, b_ks, L.eb, L.sb, sB, L.Np);
  TNX_LAUNCH_CHECK();
  CUtensorMap ma, mb;
  TNX_TRY(make_tma_map_bf16(&ma, L.sa, int64_t(batch) * OZ_S * L.Mp, L.Kp, OZ_BK, OZ_BM));
  TNX_TRY(make_tma_map_bf16(&mb, L.sb, int64_t(batch) * OZ_S * L.Np, L.Kp, OZ_BK, OZ_BN));
  const size_t smem = oz_smem_bytes();
  static DeviceSet allowed;
  TNX_CUDA(allow_smem(oz_gemm_kernel, smem, allowed));
  const int kb_all = int(L.Kp / OZ_BK);
  const int kbs = (kb_all + nsplit - 1) / nsplit;
  nsplit = (kb_all + kbs - 1) / kbs;  // no empty splits
  const int64_t items = (L.Np / OZ_BN) * (L.Mp / OZ_BM) * batch * nsplit;
  TNX_CHECK_SHAPE(items < (int64_t(1) << 30), "gemm_oz: too many tiles");
  const unsigned grid = unsigned(std::min<int64_t>(items, 152));
  // profiler family: the large products (environment updates, anchor matvecs, the gauge move's
  // X, Q and R A) apart from the narrow ones (a side of 128 or less, split K, batches)
  const int fam = (nsplit > 1 || batch > 1 || m <= 128 || n <= 128 || k <= 128) ? KF_OZ_NARROW : KF_OZ_GEMM;
  profile_mark(fam, st, true);
  oz_gemm_kernel<<<grid, OZ_THREADS, smem, st>>>(ma, mb, int(m), int(n), int(L.Kp), int(L.Mp), int(L.Np), L.ea, L.eb,
                                                 alpha, beta, C, ldc, L.flag, L.flag + 1, batch, nsplit, kbs, sC, L.part,
                                                 mask);
  TNX_LAUNCH_CHECK();
  if (nsplit > 1) {
    const int64_t mn = m * n;
    const unsigned gx = unsigned(std::min<int64_t>((mn + 255) / 256, 64));
    oz_split_reduce_kernel<<<dim3(gx, unsigned(batch)), 256, 0, st>>>(L.part, nsplit, batch, int(m), int(n), alpha,
                                                                      beta, C, ldc, sC, mask);
    TNX_LAUNCH_CHECK();
  }
  profile_mark(fam, st, false);
  profile_work(fam, 2.0 * double(m) * n * k * batch, 8.0 * batch * (double(m) * k + double(k) * n + double(m) * n));
  return TNX_OK;
}

int gemm_oz(bool ta, bool tb, int64_t m, int64_t n, int64_t k, double alpha, const double* A, int64_t lda,
            const double* B, int64_t ldb, double beta, double* C, int64_t ldc, void* ws, size_t ws_bytes,
            cudaStream_t st) {
  return gemm_oz_ex(ta, tb, m, n, k, alpha, A, lda, 0, B, ldb, 0, beta, C, ldc, 0, 1, 1, nullptr, ws, ws_bytes, st);
}

int gemm_oz_flag(void* ws, int64_t m, int64_t n, int64_t k, int** flag) {
  OzLayout L;
  oz_layout(m, n, k, 1, 1, ws, &L);
  *flag = L.flag;
  return TNX_OK;
}

}  // namespace tnx

using namespace tnx;

extern "C" {

size_t tnx_gemm_oz_workspace_bytes(int64_t m, int64_t n, int64_t k) { return gemm_oz_workspace_bytes(m, n, k); }

int tnx_gemm_oz(int trans_a, int trans_b, int64_t m, int64_t n, int64_t k, double alpha, const double* A, int64_t lda,
                const double* B, int64_t ldb, double beta, double* C, int64_t ldc, void* workspace,
                size_t workspace_bytes, void* stream) {
  TNX_CHECK_ARG(A && B && C, "null pointer");
  TNX_CHECK_ARG(m >= 0 && n >= 0 && k >= 0, "negative size");
  cudaStream_t st = as_stream(stream);
  TNX_TRY(gemm_oz(trans_a != 0, trans_b != 0, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, workspace,
                  workspace_bytes, st));
  // a bounded wait that expired inside the kernel is reported here (one 4-byte read)
  int* flag = nullptr;
  gemm_oz_flag(workspace, m, n, k, &flag);
  int h = 0;
  TNX_CUDA(cudaMemcpyAsync(&h, flag, sizeof(int), cudaMemcpyDeviceToHost, st));
  TNX_CUDA(cudaStreamSynchronize(st));
  if (h) {
    set_error("tnx_gemm_oz: a bounded wait in the tensor-core kernel expired");
    return TNX_ERR_TIMEOUT;
  }
  return TNX_OK;
}

size_t tnx_gemm_oz_batched_workspace_bytes(int64_t m, int64_t n, int64_t k, int batch, int nsplit) {
  return gemm_oz_ex_workspace_bytes(m, n, k, batch < 1 ? 1 : batch, nsplit < 1 ? 1 : nsplit);
}

int tnx_gemm_oz_batched(int trans_a, int trans_b, int64_t m, int64_t n, int64_t k, double alpha, const double* A,
                        int64_t lda, int64_t sA, const double* B, int64_t ldb, int64_t sB, double beta, double* C,
                        int64_t ldc, int64_t sC, int batch, int nsplit, const int* mask, void* workspace,
                        size_t workspace_bytes, void* stream) {
  TNX_CHECK_ARG(A && B && C, "null pointer");
  TNX_CHECK_ARG(m >= 0 && n >= 0 && k >= 0 && batch >= 1 && nsplit >= 1, "negative size, batch or split");
  cudaStream_t st = as_stream(stream);
  TNX_TRY(gemm_oz_ex(trans_a != 0, trans_b != 0, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch,
                     nsplit, mask, workspace, workspace_bytes, st));
  int* flag = nullptr;
  OzLayout L;
  oz_layout(m, n, k, batch, nsplit, workspace, &L);
  flag = L.flag;
  int h = 0;
  TNX_CUDA(cudaMemcpyAsync(&h, flag, sizeof(int), cudaMemcpyDeviceToHost, st));
  TNX_CUDA(cudaStreamSynchronize(st));
  if (h) {
    set_error("tnx_gemm_oz_batched: a bounded wait in the tensor-core kernel expired");
    return TNX_ERR_TIMEOUT;
  }
  return TNX_OK;
}

}  // extern "C"
