// Split-BF16 ("bf16x3") one-site matvec on the tcgen05 tensor cores.
//
// Each FP64 operand X is split into X_hi = bf16(X) and X_lo = bf16(X - X_hi); a product is
// taken as A_hi B_hi + A_hi B_lo + A_lo B_hi with FP32 accumulation in tensor memory, i.e.
// one BF16 GEMM over a K dimension three times as long. Relative error ~2^-16 per product.
//
// The matvec y = H_eff x of Environment.one_site_matvec (tnpy/matrix_product_state.py:411-440)
// is three steps:
//   1. T1[(w,a'),(s,c)] = sum_a L[a,(w,a')] x[a,(s,c)]        tensor cores, K = chi_l
//   2. T2[(a',s'),(c,v)] = sum_{w,s} T1 W[w,v,s,s']            CUDA cores, K = D*d, writes the
//                                                              split BF16 operand of step 3
//   3. y[(a',s'),c'] = sum_{(c,v)} T2 R[(c,v),c']             tensor cores, K = chi_r*D
// L and R are re-laid out once per site as K-major split operands (Davidson reuses them for
// every matvec of the site); x is re-laid out per matvec.
//
// GEMM kernels: one 128 x 128 output tile per CTA, or 256 x BN per pair of CTAs; 6 warps:
//   warp 0  TMA producer (cp.async.bulk.tensor, 128B swizzle, 64-wide K slabs, 4-stage ring)
//   warp 1  TMEM allocation + tcgen05.mma issue by one lane (kind::f16, BF16 in, FP32 acc)
//   warps 2-5 epilogue: tcgen05.ld of the FP32 accumulator, staged through shared memory in
//             64-column chunks, stored as FP32 or FP64 row segments
// Every mbarrier wait is bounded (~2 s of clock); on expiry the kernel raises a flag in
// global memory, stops issuing work, waits (bounded) for its own TMA copies and frees TMEM.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstring>

#include "tc_ptx.cuh"
#include "tnx_internal.cuh"
#include "wcontract.cuh"

namespace tnx {
namespace {

using namespace tc;

constexpr int BM = 128;
constexpr int BK = 64;  // 64 bf16 = 128 bytes = one swizzle atom row
constexpr int STAGES = 4;
constexpr int GEMM_THREADS = 192;

// ---------------------------------------------------------------- GEMM kernels
// Accumulator of the tile at (m0, n0) in tensor memory -> out, by warps 2 .. 5 through shared memory at stg, the
// 32 rows of a warp 64 columns at a time: in pairs of columns, whose 66-word (FP64: 132-word) row stride
// is free of conflicts, and out again as row segments of 64 columns by the same warp
constexpr int CW = 64, LD_OUT = CW + 2;                      // columns of a chunk and their row stride
constexpr uint32_t STAGING_BYTES = BM * LD_OUT * sizeof(double);  // of the four warps' chunks, in the stage ring
template <int BN, typename T>
__device__ __forceinline__ void store_tile_as(uint32_t tmem, uint8_t* stg, int m0, int n0, int M, int N,
                                              T* __restrict__ out, int64_t ldc) {
  struct alignas(2 * sizeof(T)) T2 {
    T a, b;
  };
  constexpr int LD = LD_OUT;
  const int quad = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31;  // TMEM lanes 32*quad .. 32*quad+31
  T* rows = reinterpret_cast<T*>(stg) + quad * 32 * LD;
  auto val = [](uint32_t x) {
    if constexpr (sizeof(T) == 8) return float_to_double(__uint_as_float(x));
    else return __uint_as_float(x);
  };
  const int left = M - m0 - quad * 32;  // rows of this warp inside the matrix
  const bool pairs = ldc % 2 == 0 && reinterpret_cast<uintptr_t>(out) % (2 * sizeof(T)) == 0;
#pragma unroll 1
  for (int c0 = 0; c0 < BN; c0 += CW) {
    uint32_t r[2][32];
    tmem_ld32_async(tmem + (uint32_t(quad * 32) << 16) + uint32_t(c0), r[0]);
    tmem_ld32_async(tmem + (uint32_t(quad * 32) << 16) + uint32_t(c0 + 32), r[1]);
    tmem_ld_wait();
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int j = 0; j < 32; j += 2)
        *reinterpret_cast<T2*>(rows + lane * LD + h * 32 + j) = T2{val(r[h][j]), val(r[h][j + 1])};
    __syncwarp();
    const int c = n0 + c0 + 2 * lane;
    T* dst = out + int64_t(m0 + quad * 32) * ldc + c;
    const T* src = rows + 2 * lane;
    if (pairs && c + 1 < N) {
#pragma unroll 8
      for (int i = 0; i < 32; ++i)
        if (i < left) *reinterpret_cast<T2*>(dst + i * ldc) = *reinterpret_cast<const T2*>(src + i * LD);
    } else {
      for (int i = 0; i < 32 && i < left; ++i) {
        if (c < N) dst[i * ldc] = src[i * LD];
        if (c + 1 < N) dst[i * ldc + 1] = src[i * LD + 1];
      }
    }
    __syncwarp();  // the chunk is out before the next one is staged
  }
}
template <int BN>
__device__ __forceinline__ void store_tile(uint32_t tmem, uint8_t* stg, int m0, int n0, int M, int N, void* out,
                                           int64_t ldc, int out_fp64) {
  if (out_fp64) store_tile_as<BN>(tmem, stg, m0, n0, M, N, static_cast<double*>(out), ldc);
  else store_tile_as<BN>(tmem, stg, m0, n0, M, N, static_cast<float*>(out), ldc);
}

// C[M, N] = sum_k A[m, k] B[n, k] over the three split products; A*, B* are K-major BF16
// with row pitch Kp (a multiple of 64). out: FP32 or FP64, row-major with leading dim ldc.
template <int BN>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
    bf16x3_gemm_kernel(const __grid_constant__ CUtensorMap ta_hi, const __grid_constant__ CUtensorMap ta_lo,
                       const __grid_constant__ CUtensorMap tb_hi, const __grid_constant__ CUtensorMap tb_lo,
                       int M, int N, int Kp, void* __restrict__ out, int64_t ldc, int out_fp64,
                       int* __restrict__ err_flag) {
  constexpr uint32_t A_BYTES = BM * BK * 2;
  constexpr uint32_t B_BYTES = BN * BK * 2;
  constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr uint32_t TMEM_COLS = BN < 32 ? 32 : BN;
  static_assert(STAGES * STAGE_BYTES >= STAGING_BYTES, "the epilogue stages a chunk in the ring");
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full_bar[STAGES], empty_bar[STAGES], accum_bar;
  __shared__ uint32_t tmem_base_sh;
  __shared__ int abort_sh;

  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int kblocks = Kp / BK;
  const int total = 3 * kblocks;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    mbar_init(smem_u32(&accum_bar), 1);
    abort_sh = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base_sh, 0);

  if (warp == 0) {
    // ------------------------------------------------ TMA producer
    if (lane == 0) {
      int issued = 0;
      for (int it = 0; it < total; ++it) {
        const int s = it % STAGES;
        const uint32_t ph = (it / STAGES) & 1;
        if (it >= STAGES && !mbar_wait(smem_u32(&empty_bar[s]), ph ^ 1)) {
          atomicExch(err_flag, 1);
          abort_sh = 1;
          break;
        }
        if (*((volatile int*)&abort_sh)) break;
        const int seg = it / kblocks, kb = it % kblocks;
        const CUtensorMap* ma = seg == 2 ? &ta_lo : &ta_hi;
        const CUtensorMap* mb = seg == 1 ? &tb_lo : &tb_hi;
        const uint32_t sa = base + s * STAGE_BYTES, sb = sa + A_BYTES;
        const uint32_t fb = smem_u32(&full_bar[s]);
        mbar_expect_tx(fb, STAGE_BYTES);
        tma_load_2d(sa, ma, fb, kb * BK, m0);
        tma_load_2d(sb, mb, fb, kb * BK, n0);
        ++issued;
      }
      // drain: wait (bounded) until every issued copy has landed before the CTA can exit
      for (int it = issued - STAGES < 0 ? 0 : issued - STAGES; it < issued; ++it)
        mbar_wait(smem_u32(&full_bar[it % STAGES]), (it / STAGES) & 1);
    }
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer: the whole warp runs the loop, so that descriptors
    // and addresses stay in uniform registers; one lane issues (by one lane's loop a slab took 600 clocks to
    // issue, more than its products take)
    constexpr uint32_t idesc = instr_desc_bf16(BM, BN);
    const uint32_t full0 = smem_u32(full_bar), empty0 = smem_u32(empty_bar);
    const uint64_t desc0 = smem_desc_sw128(base);
    const bool one = elect_one();
    bool ok = true;
    int s = 0;
    uint32_t ph = 0;
    for (int it = 0; it < total; ++it) {
      if (!mbar_wait(full0 + 8 * s, ph)) {
        if (one) atomicExch(err_flag, 1);
        abort_sh = 1;
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      // addresses sit in the descriptors in units of 16 bytes
      const uint64_t ad = desc0 + uint32_t(s) * (STAGE_BYTES >> 4), bd = ad + (A_BYTES >> 4);
      if (one) {
#pragma unroll
        for (int kk = 0; kk < BK / 16; ++kk)
          mma_bf16(tmem, ad + 2 * kk, bd + 2 * kk, idesc, (it > 0 || kk > 0) ? 1u : 0u);
        mma_commit(empty0 + 8 * s);
      }
      if (++s == STAGES) {
        s = 0;
        ph ^= 1;
      }
    }
    if (ok && one) mma_commit(smem_u32(&accum_bar));
  } else {
    // ------------------------------------------------ epilogue (warps 2..5)
    // The accumulator goes out in 64-column chunks through shared memory (the stage ring is free
    // once the accumulator is complete): a thread holds one row of the tile in TMEM, and storing
    // from there would write 32 rows per warp instruction; from shared memory every warp store
    // covers 32 consecutive columns of one row.
    const bool ok = mbar_wait(smem_u32(&accum_bar), 0);
    if (!ok && lane == 0) atomicExch(err_flag, 1);
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (ok) store_tile<BN>(tmem, smem_raw + (base - smem_u32(smem_raw)), m0, n0, M, N, out, ldc, out_fp64);
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
  }
}

// The same product with 256 x BN tiles by pairs of CTAs (cta_group::2): each holds its 128 rows of A and
// half of the tile's rows of B, so an SM takes in 128 + BN / 2 rows a K slab for 128 x BN products where
// the kernel above takes 128 + BN, at about 64 bytes a clock. Every output sums the same products in the
// same order as above.
//
// ST stages of SL slabs of 64; MINB CTAs on an SM. What bounded the kernel was neither: waiting for a stage,
// issuing its four products and the commit took the issuing lane 600 clocks a slab, whose products take 256
// (BN = 128) to 512. Run by the whole warp with uniform operands, and with two slabs a stage, it is
// below that; two CTAs on an SM hide it too, and one's stores run beside the other's products where tiles
// outnumber the SMs. chi = 1024: 5120 x 2048 x 1024 89 us by single CTAs with 128 x 256 tiles, 54 us
// with <192, 3, 1, 2> here; 2048 x 1024 x 5120 85 us with 128 x 128 tiles, 52 us with <128, 4, 2, 1>. The
// epilogue's row segments in place of element by element made 8 us of each.
template <int BN, int ST, int SL, int MINB>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, MINB)
    bf16x3_pair_kernel(const __grid_constant__ CUtensorMap ta_hi, const __grid_constant__ CUtensorMap ta_lo,
                       const __grid_constant__ CUtensorMap tb_hi, const __grid_constant__ CUtensorMap tb_lo,
                       int M, int N, int Kp, int tiles_n, void* __restrict__ out, int64_t ldc, int out_fp64,
                       int* __restrict__ err_flag) {
  constexpr uint32_t A_BYTES = BM * BK * 2;
  constexpr uint32_t B_BYTES = BN / 2 * BK * 2;
  constexpr uint32_t SLAB_BYTES = A_BYTES + B_BYTES, STAGE_BYTES = SL * SLAB_BYTES;
  constexpr uint32_t TMEM_COLS = BN <= 128 ? 128 : 256;
  static_assert(ST * STAGE_BYTES >= STAGING_BYTES, "the epilogue stages a chunk in the ring");
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full_bar[ST], empty_bar[ST], accum_bar;  // full: rank 0's, for both
  __shared__ uint32_t tmem_base_sh;
  __shared__ int abort_sh;

  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int tile = blockIdx.x >> 1;
  const int m0 = (tile / tiles_n * 2 + int(rank)) * BM, n0 = tile % tiles_n * BN;
  const int kblocks = Kp / BK;
  const int ksteps = (kblocks + SL - 1) / SL, total = 3 * ksteps;  // stages of SL slabs; the last of a product may be short

  if (threadIdx.x == 0) {
    for (int s = 0; s < ST; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    mbar_init(smem_u32(&accum_bar), 1);
    abort_sh = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers and tensor memory are there
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base_sh, 0);

  if (warp == 0) {
    // ------------------------------------------------ TMA producer of this CTA's rows
    if (lane == 0) {
      int issued = 0, s = 0;
      uint32_t ph = 0;
      const uint32_t full0 = smem_u32(full_bar), empty0 = smem_u32(empty_bar), fb0 = rank_addr(full0, 0);
      const int nb0 = n0 + int(rank) * (BN / 2);
      bool ok = true;
      for (int seg = 0; seg < 3 && ok; ++seg) {
        const CUtensorMap* ma = seg == 2 ? &ta_lo : &ta_hi;
        const CUtensorMap* mb = seg == 1 ? &tb_lo : &tb_hi;
        for (int kb = 0; kb < kblocks; kb += SL) {
          if ((issued >= ST && !mbar_wait(empty0 + 8 * s, ph ^ 1)) || *((volatile int*)&abort_sh)) {
            if (!*((volatile int*)&abort_sh)) atomicExch(err_flag, 1);
            abort_sh = 1;
            ok = false;
            break;
          }
          const uint32_t sa = base + s * STAGE_BYTES;
          const int slabs = kblocks - kb < SL ? kblocks - kb : SL;
          if (rank == 0) mbar_expect_tx(full0 + 8 * s, 2 * SLAB_BYTES * slabs);
#pragma unroll
          for (int i = 0; i < SL; ++i)
            if (i < slabs) {
              tma_load_2d_pair(sa + i * SLAB_BYTES, ma, fb0 + 8 * s, (kb + i) * BK, m0);
              tma_load_2d_pair(sa + i * SLAB_BYTES + A_BYTES, mb, fb0 + 8 * s, (kb + i) * BK, nb0);
            }
          ++issued;
          if (++s == ST) {
            s = 0;
            ph ^= 1;
          }
        }
      }
      // drain: wait (bounded) until every copy that rank 0 counts has landed before the CTAs can exit
      if (rank == 0)
        for (int it = issued - ST < 0 ? 0 : issued - ST; it < issued; ++it)
          mbar_wait(smem_u32(&full_bar[it % ST]), (it / ST) & 1);
    }
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer (rank 0). The whole warp runs the loop, so that
    // descriptors and addresses stay in uniform registers; one lane issues
    if (rank == 0) {
      constexpr uint32_t idesc = instr_desc_bf16(2 * BM, BN);
      const uint32_t full0 = smem_u32(full_bar), empty0 = smem_u32(empty_bar);
      const uint64_t desc0 = smem_desc_sw128(base);
      const bool one = elect_one();
      bool ok = true;
      int s = 0, left = kblocks;
      uint32_t ph = 0;
      for (int it = 0; it < total; ++it) {
        if (!mbar_wait(full0 + 8 * s, ph)) {
          if (one) atomicExch(err_flag, 1);
          abort_sh = 1;
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        // addresses sit in the descriptors in units of 16 bytes
        const uint64_t ad = desc0 + uint32_t(s) * (STAGE_BYTES >> 4), bd = ad + (A_BYTES >> 4);
        if (one) {
#pragma unroll
          for (int i = 0; i < SL; ++i)
            if (i < left)
#pragma unroll
              for (int kk = 0; kk < BK / 16; ++kk)
                mma_bf16_pair(tmem, ad + i * (SLAB_BYTES >> 4) + 2 * kk, bd + i * (SLAB_BYTES >> 4) + 2 * kk, idesc,
                              (it > 0 || i > 0 || kk > 0) ? 1u : 0u);
          mma_commit_pair(empty0 + 8 * s);
        }
        left = left > SL ? left - SL : kblocks;
        if (++s == ST) {
          s = 0;
          ph ^= 1;
        }
      }
      if (ok && one) mma_commit_pair(smem_u32(&accum_bar));
    }
  } else {
    // ------------------------------------------------ epilogue of this CTA's rows (warps 2..5)
    const bool ok = mbar_wait(smem_u32(&accum_bar), 0);
    if (!ok && lane == 0) atomicExch(err_flag, 1);
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (ok) store_tile<BN>(tmem, smem_raw + (base - smem_u32(smem_raw)), m0, n0, M, N, out, ldc, out_fp64);
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  cluster_sync_all();  // nothing reads the other CTA's shared or tensor memory any more
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
  cluster_sync_all();
}

// ---------------------------------------------------------------- operand preparation
// hi = v rounded to BF16, lo = v - hi (exact in FP64) rounded to BF16, as bit patterns: integer
// arithmetic on the 53-bit significand, because a conversion or an addition holds the FP64 pipe for
// 64 clocks a warp. Round to nearest even, subnormal results and overflow included; Inf and NaN as
// the conversions give them (lo NaN).
__device__ __forceinline__ uint32_t round_bf16(uint64_t sig, int e, uint32_t sign) {
  // sign * sig * 2^e, sig < 2^54, to BF16
  if (sig == 0) return sign << 15;
  const int p = 63 - __clzll(static_cast<long long>(sig));
  int ef = e + p + 127;                  // exponent field of a normal result
  int drop = ef > 0 ? p - 7 : p - 6 - ef;  // bits below the last kept one; a subnormal result keeps fewer
  uint64_t q;
  if (drop <= 0) {
    q = sig << -drop;  // -drop <= 7
  } else if (drop > 54) {
    q = 0;
  } else {
    const uint64_t half = (1ull << (drop - 1)) - 1 + ((sig >> drop) & 1);
    q = (sig + half) >> drop;
  }
  // q carries the implicit bit of a normal result, which adds one to the exponent field below
  const uint32_t r = ef > 0 ? (uint32_t(ef - 1) << 7) + uint32_t(q) : uint32_t(q);
  return (sign << 15) | (r < 0x7f80u ? r : 0x7f80u);
}
__device__ __forceinline__ void split_bf16(double v, uint32_t& hi, uint32_t& lo) {
  const uint64_t u = static_cast<uint64_t>(__double_as_longlong(v));
  const uint32_t sign = uint32_t(u >> 63);
  const int eb = int(u >> 52) & 0x7ff;
  const uint64_t m = u & ((1ull << 52) - 1);
  if (eb - 896 < 8 || eb - 896 >= 254) {  // near or outside BF16's normal range
    if (eb == 2047) {
      hi = m ? 0x7fffu : (sign << 15) | 0x7f80u;
      lo = 0x7fffu;
      return;
    }
    const uint64_t sig = eb ? m | (1ull << 52) : m;
    const int e = (eb ? eb : 1) - 1075;
    hi = round_bf16(sig, e, sign);
    if ((hi & 0x7fffu) == 0x7f80u) {  // overflow: v - Inf
      lo = ((sign ^ 1u) << 15) | 0x7f80u;
      return;
    }
    // hi as an integer multiple of 2^e (its last bit is at 2^-133 or above, e may be far below)
    const int hf = int(hi >> 7) & 0xff;
    const uint64_t hs = (hi & 0x7fu) | (hf ? 0x80u : 0u);
    const int he = (hf ? hf : 1) - 134 - e;  // hi = hs 2^(he + e); hs == 0 where he is out of range
    const uint64_t hv = hs ? hs << he : 0;
    lo = sig >= hv ? round_bf16(sig - hv, e, sign) : round_bf16(hv - sig, e, sign ^ 1u);
    return;
  }
  // normal hi: the upper word holds its 8 bits and the half's, the lower one only breaks ties
  const uint32_t lw = uint32_t(u), hw = (uint32_t(u >> 32) & 0xfffffu) | 0x100000u;
  const uint32_t q = (hw + 0xfffu + (((hw >> 13) & 1u) | (lw != 0 ? 1u : 0u))) >> 13;  // 128 .. 256
  hi = (sign << 15) | ((uint32_t(eb - 897) << 7) + q);
  // v - hi = d 2^(eb - 1075), |d| <= 2^44; its upper 32 bits (t, below them a sticky bit) round to 8 where they
  // hold 10 and more and the result is normal
  const uint32_t dh = hw - (q << 13), neg = dh >> 31;
  const uint64_t d = (uint64_t(dh) << 32) | lw, a = neg ? 0 - d : d;
  const uint32_t al = uint32_t(a), ah = uint32_t(a >> 32), t = __funnelshift_l(al, ah, 19);
  const int p = 31 - __clz(int(t)), ef = eb - 1075 + p + 13 + 127;
  if (p >= 9 && ef > 0) {
    const int drop = p - 7;
    const uint32_t r = (t + (1u << (drop - 1)) - 1u + (((t >> drop) & 1u) | ((al << 19) != 0 ? 1u : 0u))) >> drop;
    lo = ((sign ^ neg) << 15) | ((uint32_t(ef - 1) << 7) + r);
    return;
  }
  lo = a == 0 ? 0 : round_bf16(a, eb - 1075, sign ^ neg);  // v - hi = +0
}
__device__ __forceinline__ void split_bf16(float v, uint32_t& hi, uint32_t& lo) {
  const __nv_bfloat16 h = __float2bfloat16_rn(v);
  hi = __bfloat16_as_ushort(h);
  lo = __bfloat16_as_ushort(__float2bfloat16_rn(v - __bfloat162float(h)));
}

// dst_hi/lo[c][r] (row pitch ldp, even) = split(src[r][c]) for r < rows; zeros for rows <= r < ldp.
// src is row-major rows x cols. Bound by memory (8 bytes read, 4 written an element) once the
// split stays off the FP64 pipe: L, R and x of a chi = 1024 site 101 us with conversions, 58 us with 64-bit
// integers, 53 us with 32-bit ones.
template <typename T>
__global__ void __launch_bounds__(256) split_transpose_kernel(const T* __restrict__ src, int64_t rows, int64_t cols,
                                                             __nv_bfloat16* __restrict__ hi,
                                                             __nv_bfloat16* __restrict__ lo, int64_t ldp) {
  __shared__ T tile[64][33];
  const int64_t r0 = int64_t(blockIdx.y) * 64, c0 = int64_t(blockIdx.x) * 32;
  const int tx = threadIdx.x, ty = threadIdx.y;
  T x[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int64_t r = r0 + ty + 8 * i, c = c0 + tx;
    x[i] = (r < rows && c < cols) ? src[r * cols + c] : T(0);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) tile[ty + 8 * i][tx] = x[i];
  __syncthreads();
  const int64_t r = r0 + 2 * tx;
  if (r >= ldp) return;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int64_t c = c0 + ty + 8 * i;
    if (c >= cols) continue;
    uint32_t h0, l0, h1, l1;
    split_bf16(tile[2 * tx][ty + 8 * i], h0, l0);
    split_bf16(tile[2 * tx + 1][ty + 8 * i], h1, l1);
    *reinterpret_cast<uint32_t*>(hi + c * ldp + r) = h0 | h1 << 16;
    *reinterpret_cast<uint32_t*>(lo + c * ldp + r) = l0 | l1 << 16;
  }
}

// dst_hi/lo[r][c] (row pitch ldp) = split(src[r][c]), zeros for cols <= c < ldp
__global__ void split_pad_kernel(const double* __restrict__ src, int64_t rows, int64_t cols,
                                 __nv_bfloat16* __restrict__ hi, __nv_bfloat16* __restrict__ lo, int64_t ldp) {
  for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < rows * ldp;
       e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t r = e / ldp, c = e % ldp;
    uint32_t h, l;
    split_bf16(c < cols ? src[r * cols + c] : 0.0, h, l);
    hi[e] = __ushort_as_bfloat16(uint16_t(h));
    lo[e] = __ushort_as_bfloat16(uint16_t(l));
  }
}

// zero the padding columns [k0, ldp) of a rows x ldp bf16 pair
__global__ void zero_pad_kernel(__nv_bfloat16* __restrict__ hi, __nv_bfloat16* __restrict__ lo, int64_t rows,
                                int64_t k0, int64_t ldp) {
  const int64_t w = ldp - k0;
  for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < rows * w;
       e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t r = e / w, c = k0 + e % w;
    hi[r * ldp + c] = __float2bfloat16_rn(0.f);
    lo[r * ldp + c] = __float2bfloat16_rn(0.f);
  }
}

// ---------------------------------------------------------------- host side
// 2-D map over a K-major bf16 matrix rows x ldp (K innermost), box {64, box_rows}, 128B swizzle
int make_map(CUtensorMap* map, const void* ptr, int64_t rows, int64_t ldp, int box_rows) {
  return make_tma_map_bf16(map, ptr, rows, ldp, BK, box_rows);
}

template <int BN>
size_t gemm_smem_bytes() {
  return size_t(STAGES) * (BM * BK * 2 + BN * BK * 2) + 1024;
}

template <int BN>
int launch_gemm(const __nv_bfloat16* a_hi, const __nv_bfloat16* a_lo, const __nv_bfloat16* b_hi,
                const __nv_bfloat16* b_lo, int M, int N, int Kp, void* out, int64_t ldc, bool out_fp64,
                int* err_flag, cudaStream_t st, int64_t k_real = -1) {
  CUtensorMap mah, mal, mbh, mbl;
  TNX_TRY(make_map(&mah, a_hi, M, Kp, BM));
  TNX_TRY(make_map(&mal, a_lo, M, Kp, BM));
  TNX_TRY(make_map(&mbh, b_hi, N, Kp, BN));
  TNX_TRY(make_map(&mbl, b_lo, N, Kp, BN));
  const size_t smem = gemm_smem_bytes<BN>();
  static DeviceSet allowed;
  TNX_CUDA(allow_smem(bf16x3_gemm_kernel<BN>, smem, allowed));
  dim3 grid(unsigned((N + BN - 1) / BN), unsigned((M + BM - 1) / BM));
  profile_mark(KF_TC_GEMM, st, true);
  bf16x3_gemm_kernel<BN><<<grid, GEMM_THREADS, smem, st>>>(mah, mal, mbh, mbl, M, N, Kp, out, ldc,
                                                           out_fp64 ? 1 : 0, err_flag);
  profile_mark(KF_TC_GEMM, st, false);
  // algorithmic work: one product of the unsplit operands (2 M N K flops)
  profile_work(KF_TC_GEMM, 2.0 * M * N * double(k_real < 0 ? Kp : k_real),
               2.0 * 2.0 * (double(M) + N) * Kp * 3 + double(M) * N * (out_fp64 ? 8 : 4));
  TNX_LAUNCH_CHECK();
  return TNX_OK;
}

template <int BN, int ST, int SL, int MINB>
int launch_pair(const __nv_bfloat16* a_hi, const __nv_bfloat16* a_lo, const __nv_bfloat16* b_hi,
                const __nv_bfloat16* b_lo, int M, int N, int Kp, void* out, int64_t ldc, bool out_fp64, int* err_flag,
                cudaStream_t st, int64_t k_real) {
  CUtensorMap mah, mal, mbh, mbl;
  TNX_TRY(make_map(&mah, a_hi, M, Kp, BM));
  TNX_TRY(make_map(&mal, a_lo, M, Kp, BM));
  TNX_TRY(make_map(&mbh, b_hi, N, Kp, BN / 2));
  TNX_TRY(make_map(&mbl, b_lo, N, Kp, BN / 2));
  const size_t smem = size_t(ST) * SL * (BM + BN / 2) * BK * 2 + 1024;
  static DeviceSet allowed;
  TNX_CUDA((allow_smem(bf16x3_pair_kernel<BN, ST, SL, MINB>, smem, allowed)));
  const int tn = (N + BN - 1) / BN, tm = (M + 2 * BM - 1) / (2 * BM);
  profile_mark(KF_TC_GEMM, st, true);
  bf16x3_pair_kernel<BN, ST, SL, MINB><<<2 * tn * tm, GEMM_THREADS, smem, st>>>(mah, mal, mbh, mbl, M, N, Kp, tn, out, ldc,
                                                                            out_fp64 ? 1 : 0, err_flag);
  profile_mark(KF_TC_GEMM, st, false);
  profile_work(KF_TC_GEMM, 2.0 * M * N * double(k_real),
               2.0 * 2.0 * (double(M) + N) * Kp * 3 + double(M) * N * (out_fp64 ? 8 : 4));
  TNX_LAUNCH_CHECK();
  return TNX_OK;
}

// C = A B^T in the split products by variant v: 0 one CTA a tile of 128 x 128, 1 - 3 pairs with 256 x 128, 192, 256
int split_gemm(int v, const __nv_bfloat16* a_hi, const __nv_bfloat16* a_lo, const __nv_bfloat16* b_hi,
               const __nv_bfloat16* b_lo, int64_t M, int64_t N, int64_t Kp, void* out, int64_t ldc, bool out_fp64,
               int* err_flag, cudaStream_t st, int64_t k_real) {
  const int m = int(M), n = int(N), k = int(Kp);
  switch (v) {
    case 0: return launch_gemm<128>(a_hi, a_lo, b_hi, b_lo, m, n, k, out, ldc, out_fp64, err_flag, st, k_real);
    case 1: return launch_pair<128, 4, 2, 1>(a_hi, a_lo, b_hi, b_lo, m, n, k, out, ldc, out_fp64, err_flag, st, k_real);
    case 2: return launch_pair<192, 3, 1, 2>(a_hi, a_lo, b_hi, b_lo, m, n, k, out, ldc, out_fp64, err_flag, st, k_real);
    default: return launch_pair<256, 3, 2, 1>(a_hi, a_lo, b_hi, b_lo, m, n, k, out, ldc, out_fp64, err_flag, st, k_real);
  }
}
constexpr int SPLIT_VARIANTS = 4;
// Variant where no timing is possible or wanted: rows taken in by the busiest SM, (tiles a SM or pair) x
// (rows a slab)
int split_rule(int64_t M, int64_t N) {
  const int64_t m1 = (M + 127) / 128, m2 = (M + 255) / 256;
  const int64_t sms = 152;
  auto waves = [](int64_t tiles, int64_t slots) { return (tiles + slots - 1) / slots; };
  const int64_t cost[SPLIT_VARIANTS] = {waves(m1 * ((N + 127) / 128), sms) * 256,
                                        waves(m2 * ((N + 127) / 128), sms / 2) * 192,
                                        waves(m2 * ((N + 191) / 192), sms / 2) * 224,
                                        waves(m2 * ((N + 255) / 256), sms / 2) * 256};
  int best = 0;
  for (int v = 1; v < SPLIT_VARIANTS; ++v)
    if (cost[v] < cost[best]) best = v;
  return best;
}

inline int64_t pad64(int64_t k) { return (k + 63) / 64 * 64; }

struct MixedLayout {
  int64_t K1p, K3p, M1, N1, M3, N3;
  __nv_bfloat16 *a1h, *a1l, *b1h, *b1l, *a3h, *a3l, *b3h, *b3l;
  float* T1;
  int* flag;
};

size_t mixed_layout(int64_t chi_l, int64_t d, int64_t chi_r, int64_t dl, int64_t dr, void* base, MixedLayout* L) {
  MixedLayout m;
  m.K1p = pad64(chi_l);
  m.K3p = pad64(chi_r * dr);
  m.M1 = dl * chi_l;
  m.N1 = d * chi_r;
  m.M3 = chi_l * d;
  m.N3 = chi_r;
  size_t off = 0;
  auto take = [&](size_t bytes) { size_t o = off; off += align_up(bytes, 1024); return o; };
  size_t o1 = take(m.M1 * m.K1p * 2), o2 = take(m.M1 * m.K1p * 2), o3 = take(m.N1 * m.K1p * 2),
         o4 = take(m.N1 * m.K1p * 2), o5 = take(m.M3 * m.K3p * 2), o6 = take(m.M3 * m.K3p * 2),
         o7 = take(m.N3 * m.K3p * 2), o8 = take(m.N3 * m.K3p * 2), o9 = take(m.M1 * m.N1 * 4), o10 = take(256);
  if (base && L) {
    char* b = static_cast<char*>(base);
    m.a1h = reinterpret_cast<__nv_bfloat16*>(b + o1);
    m.a1l = reinterpret_cast<__nv_bfloat16*>(b + o2);
    m.b1h = reinterpret_cast<__nv_bfloat16*>(b + o3);
    m.b1l = reinterpret_cast<__nv_bfloat16*>(b + o4);
    m.a3h = reinterpret_cast<__nv_bfloat16*>(b + o5);
    m.a3l = reinterpret_cast<__nv_bfloat16*>(b + o6);
    m.b3h = reinterpret_cast<__nv_bfloat16*>(b + o7);
    m.b3l = reinterpret_cast<__nv_bfloat16*>(b + o8);
    m.T1 = reinterpret_cast<float*>(b + o9);
    m.flag = reinterpret_cast<int*>(b + o10);
    *L = m;
  }
  return off + 1024;  // slack for aligning the base
}

void* align1024(void* p) {
  return reinterpret_cast<void*>((reinterpret_cast<uintptr_t>(p) + 1023) & ~uintptr_t(1023));
}

dim3 tgrid(int64_t rows, int64_t cols) {
  return dim3(unsigned((cols + 31) / 32), unsigned((rows + 63) / 64));
}

}  // namespace

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeFn get_encode() {
  static EncodeFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return reinterpret_cast<EncodeFn>(p);
    return static_cast<EncodeFn>(nullptr);
  }();
  return fn;
}

int make_tma_map_bf16(CUtensorMap* map, const void* ptr, int64_t rows, int64_t ldp, int box_k, int box_rows) {
  EncodeFn enc = get_encode();
  if (!enc) {
    set_error("cuTensorMapEncodeTiled unavailable");
    return TNX_ERR_CUDA;
  }
  if ((reinterpret_cast<uintptr_t>(ptr) & 15) != 0 || (ldp * 2) % 16 != 0 || (box_k != 64 && box_k != 32)) {
    set_error("TMA operand misaligned");
    return TNX_ERR_INVALID_ARG;
  }
  cuuint64_t dims[2] = {cuuint64_t(ldp), cuuint64_t(rows)};
  cuuint64_t strides[1] = {cuuint64_t(ldp * 2)};
  cuuint32_t box[2] = {cuuint32_t(box_k), cuuint32_t(box_rows)};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, box_k == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d)", int(r));
    return TNX_ERR_CUDA;
  }
  return TNX_OK;
}

bool mixed_supported(int64_t chi_l, int64_t d, int64_t chi_r, int64_t dl, int64_t dr) {
  return chi_l >= 16 && chi_r >= 16 && dl * d <= 64 && dr * d <= 64 && dl * chi_l < (1 << 30);
}

size_t matvec1_bf16x3_scratch_bytes(int64_t chi_l, int64_t d, int64_t chi_r, int64_t dl, int64_t dr) {
  return mixed_layout(chi_l, d, chi_r, dl, dr, nullptr, nullptr);
}

// Per-site preparation: split + transpose L and R, zero the padding of the T2 operand.
int mixed_prepare(const double* L, const double* R, int64_t chi_l, int64_t d, int64_t chi_r, int64_t dl, int64_t dr,
                  void* scratch, cudaStream_t st) {
  MixedLayout m;
  mixed_layout(chi_l, d, chi_r, dl, dr, align1024(scratch), &m);
  dim3 tb(32, 8);
  // A1[(w a')][a] = L[a][(w a')]: src rows = chi_l, cols = dl*chi_l, pitch K1p
  split_transpose_kernel<double><<<tgrid(m.K1p, m.M1), tb, 0, st>>>(L, chi_l, m.M1, m.a1h, m.a1l, m.K1p);
  TNX_LAUNCH_CHECK();
  // B3[c'][(c v)] = R[(c v)][c']: src rows = chi_r*dr, cols = chi_r, pitch K3p
  split_transpose_kernel<double><<<tgrid(m.K3p, m.N3), tb, 0, st>>>(R, chi_r * dr, chi_r, m.b3h, m.b3l, m.K3p);
  TNX_LAUNCH_CHECK();
  if (m.K3p > chi_r * dr) {
    zero_pad_kernel<<<152, 256, 0, st>>>(m.a3h, m.a3l, m.M3, chi_r * dr, m.K3p);
    TNX_LAUNCH_CHECK();
  }
  TNX_CUDA(cudaMemsetAsync(m.flag, 0, sizeof(int), st));
  return TNX_OK;
}

// One matvec with prepared L / R operands; x and y FP64 or FP32 (T).
template <typename T>
int mixed_apply_t(const double* W, const T* x, T* y, int64_t chi_l, int64_t d, int64_t chi_r, int64_t dl,
                  int64_t dr, void* scratch, cudaStream_t st) {
  MixedLayout m;
  mixed_layout(chi_l, d, chi_r, dl, dr, align1024(scratch), &m);
  dim3 tb(32, 8);
  // B1[(s c)][a] = x[a][(s c)]
  split_transpose_kernel<T><<<tgrid(m.K1p, m.N1), tb, 0, st>>>(x, chi_l, m.N1, m.b1h, m.b1l, m.K1p);
  TNX_LAUNCH_CHECK();
  // step 1: T1 (FP32) = A1 . B1^T; tiles autotuned per shape
  {
    auto run = [&](int v) -> int {
      return split_gemm(v, m.a1h, m.a1l, m.b1h, m.b1l, m.M1, m.N1, m.K1p, m.T1, m.N1, false, m.flag, st, chi_l);
    };
    TNX_TRY(autotuned(TuneKey{3, m.M1, m.N1, m.K1p, 0, 0}, SPLIT_VARIANTS, split_rule(m.M1, m.N1), m.N1 >= 256, st, run));
  }
  // step 2: MPO contraction into the split A3 operand, [(a',s')][(c,v)] with row pitch K3p (wcontract.cuh)
  TNX_TRY((wc::launch_left<float>(m.T1, 0, W, 0, wc::OutSplit{m.a3h, m.a3l}, 0, chi_l, d, chi_r, dl, dr, m.K3p, 1,
                                  nullptr, st)));
  // step 3: y = A3 . B3^T (FP32 accumulators written as T); tiles autotuned per shape
  {
    auto run = [&](int v) -> int {
      return split_gemm(v, m.a3h, m.a3l, m.b3h, m.b3l, m.M3, m.N3, m.K3p, y, m.N3, sizeof(T) == 8, m.flag, st,
                        chi_r * dr);
    };
    TNX_TRY(autotuned(TuneKey{3, m.M3, m.N3, m.K3p, int64_t(sizeof(T)), 0}, SPLIT_VARIANTS, split_rule(m.M3, m.N3),
                      m.N3 >= 256, st, run));
  }
  return TNX_OK;
}

int mixed_apply(const double* W, const double* x, double* y, int64_t chi_l, int64_t d, int64_t chi_r, int64_t dl,
                int64_t dr, void* scratch, cudaStream_t st) {
  return mixed_apply_t<double>(W, x, y, chi_l, d, chi_r, dl, dr, scratch, st);
}

int mixed_apply_f32(const double* W, const float* x, float* y, int64_t chi_l, int64_t d, int64_t chi_r, int64_t dl,
                    int64_t dr, void* scratch, cudaStream_t st) {
  return mixed_apply_t<float>(W, x, y, chi_l, d, chi_r, dl, dr, scratch, st);
}

int mixed_flag(void* scratch, int64_t chi_l, int64_t d, int64_t chi_r, int64_t dl, int64_t dr, int** flag) {
  MixedLayout m;
  mixed_layout(chi_l, d, chi_r, dl, dr, align1024(scratch), &m);
  *flag = m.flag;
  return TNX_OK;
}

int matvec1_bf16x3(const double* L, const double* W, const double* R, const double* x, double* y, int64_t chi_l,
                   int64_t d, int64_t chi_r, int64_t dl, int64_t dr, void* scratch, size_t scratch_bytes,
                   cudaStream_t st) {
  if (!mixed_supported(chi_l, d, chi_r, dl, dr)) {
    set_error("split-BF16 matvec needs chi_l, chi_r >= 16 (got %lld, %lld)", (long long)chi_l, (long long)chi_r);
    return TNX_ERR_UNSUPPORTED;
  }
  if (scratch_bytes < matvec1_bf16x3_scratch_bytes(chi_l, d, chi_r, dl, dr) || !scratch) {
    set_error("split-BF16 matvec: scratch too small");
    return TNX_ERR_WORKSPACE;
  }
  TNX_TRY(mixed_prepare(L, R, chi_l, d, chi_r, dl, dr, scratch, st));
  return mixed_apply(W, x, y, chi_l, d, chi_r, dl, dr, scratch, st);
}


}  // namespace tnx

using namespace tnx;

extern "C" {

size_t tnx_gemm_bf16x3_workspace_bytes(int64_t m, int64_t n, int64_t k) {
  const int64_t kp = pad64(k);
  return 2 * align_up(size_t(m * kp * 2), 1024) + 2 * align_up(size_t(n * kp * 2), 1024) + 2048;
}

int tnx_gemm_bf16x3(int64_t m, int64_t n, int64_t k, const double* A, const double* B, double* C,
                    void* workspace, size_t workspace_bytes, void* stream) {
  TNX_CHECK_ARG(A && B && C, "null pointer");
  TNX_CHECK_ARG(m > 0 && n > 0 && k > 0, "non-positive size");
  TNX_CHECK_SHAPE(m < (1 << 30) && n < (1 << 30) && k < (1 << 28), "size too large");
  size_t need = tnx_gemm_bf16x3_workspace_bytes(m, n, k);
  if (workspace_bytes < need || !workspace) {
    set_error("tnx_gemm_bf16x3: workspace %zu bytes < required %zu", workspace_bytes, need);
    return TNX_ERR_WORKSPACE;
  }
  cudaStream_t st = as_stream(stream);
  const int64_t kp = pad64(k);
  char* b = static_cast<char*>(align1024(workspace));
  auto* ah = reinterpret_cast<__nv_bfloat16*>(b);
  auto* al = reinterpret_cast<__nv_bfloat16*>(b + align_up(size_t(m * kp * 2), 1024));
  auto* bh = reinterpret_cast<__nv_bfloat16*>(b + 2 * align_up(size_t(m * kp * 2), 1024));
  auto* bl = reinterpret_cast<__nv_bfloat16*>(b + 2 * align_up(size_t(m * kp * 2), 1024) +
                                              align_up(size_t(n * kp * 2), 1024));
  int* flag = reinterpret_cast<int*>(b + 2 * align_up(size_t(m * kp * 2), 1024) +
                                     2 * align_up(size_t(n * kp * 2), 1024));
  TNX_CUDA(cudaMemsetAsync(flag, 0, sizeof(int), st));
  split_pad_kernel<<<152 * 4, 256, 0, st>>>(A, m, k, ah, al, kp);
  TNX_LAUNCH_CHECK();
  split_pad_kernel<<<152 * 4, 256, 0, st>>>(B, n, k, bh, bl, kp);
  TNX_LAUNCH_CHECK();
  TNX_TRY(split_gemm(split_rule(m, n), ah, al, bh, bl, m, n, kp, C, n, true, flag, st, k));
  int host_flag = 0;
  TNX_CUDA(cudaMemcpyAsync(&host_flag, flag, sizeof(int), cudaMemcpyDeviceToHost, st));
  TNX_CUDA(cudaStreamSynchronize(st));
  if (host_flag) {
    set_error("tnx_gemm_bf16x3: a bounded device wait expired");
    return TNX_ERR_TIMEOUT;
  }
  return TNX_OK;
}

}  // extern "C"
