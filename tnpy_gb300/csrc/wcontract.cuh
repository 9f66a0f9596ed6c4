// The MPO step between the two GEMMs of a matvec or an environment update, for one site or for
// stacked chains (blockIdx.y = chain).
//
//   left  T2[(a',s'),(c,v)] = sum_{w,s} T1[(w,a'),(s,c)] W[w,v,s,s']
//   right T2[(a,w),(s',c')] = sum_{v,s} T1[(a,s),(v,c')] W[w,v,s,s']
//
// A dense W costs (dl d)(dr d) FMAs per (a', c) fibre: 1.05e8 at chi = 1024, D = 5, which the FP64
// pipe (2 FMAs per clock and SM) turns into 170 us against 25 us for the bytes. The MPOs of spin
// chains are mostly zeros (12 of 100 entries for XXZ), so every output keeps a list of its
// nonzero coefficients and runs over those only, in the dense order: the result is bit for bit
// the dense one, because adding a finite value times zero to the sum changes nothing; a tile
// that holds Inf or NaN takes the dense sum, where 0 * Inf has to give NaN.
//
// A lane owns one fibre and reads its inputs coalesced along c, all of them in flight at once;
// its shared-memory column only makes them indexable, so the loop needs no barrier. The left
// form's outputs, strided by dr, go out through the warp's shared memory as contiguous rows, in
// pairs where they lie aligned. Instructions bound it: chi = 1024, D = 5, left form: 300 us (FP64) with a dense sum
// over per-thread arrays in local memory, 69 us with bit masks and single outputs, 60 us so; 100, 46 and 35 us
// for the split-BF16 operand.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "tnx_internal.cuh"

namespace tnx {
namespace wc {

__device__ __forceinline__ bool not_finite(double x) {
  return (static_cast<unsigned long long>(__double_as_longlong(x)) & 0x7ff0000000000000ull) == 0x7ff0000000000000ull;
}
__device__ __forceinline__ bool not_finite(float x) { return (__float_as_uint(x) & 0x7f800000u) == 0x7f800000u; }

__device__ __forceinline__ bool nonzero(double x) { return (__double_as_longlong(x) << 1) != 0; }
__device__ __forceinline__ bool nonzero(float x) { return (__float_as_uint(x) << 1) != 0u; }

// where an output goes: FP64, or the split-BF16 operand (hi, lo)
struct OutF64 {
  double* p;
  __device__ void at(int64_t i, double v) const { p[i] = v; }
  // outputs i, i + 1 with even i
  __device__ bool aligned() const { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
  __device__ void two(int64_t i, const double* v) const {
    *reinterpret_cast<double2*>(p + i) = *reinterpret_cast<const double2*>(v);
  }
};
struct OutSplit {
  __nv_bfloat16 *hi, *lo;
  __device__ void at(int64_t i, float v) const {
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    hi[i] = h;
    lo[i] = __float2bfloat16_rn(v - __bfloat162float(h));
  }
  __device__ bool aligned() const {
    return ((reinterpret_cast<uintptr_t>(hi) | reinterpret_cast<uintptr_t>(lo)) & 3) == 0;
  }
  __device__ void two(int64_t i, const float* v) const {
    const float2 x = *reinterpret_cast<const float2*>(v);
    const __nv_bfloat162 h = __float22bfloat162_rn(x);
    *reinterpret_cast<__nv_bfloat162*>(hi + i) = h;
    *reinterpret_cast<__nv_bfloat162*>(lo + i) =
        __float22bfloat162_rn(make_float2(x.x - __low2float(h), x.y - __high2float(h)));
  }
};

// Shared memory of a CTA of nw warps: offsets [64] of the inputs, lengths [64] of the lists, coefficients [nout][nin]
// with their inputs' places, and per warp the inputs [nin][32] and (left form) the outputs [d][32][dr]; nin,
// nout <= 64
__host__ __device__ constexpr int list_len(int nin, int nout) { return (nin * nout + 7) / 8 * 8; }
template <typename T, bool LEFT>
__host__ __device__ constexpr size_t smem_bytes(int nin, int nout, int nw) {
  return 64 * 12 + (sizeof(T) + 2) * size_t(list_len(nin, nout)) +
         sizeof(T) * size_t(nw) * 32 * (nin + (LEFT ? nout : 0));
}

template <typename T, bool LEFT>
struct Smem {
  int64_t* off;
  int* cnt;
  T *w, *in, *out;
  uint16_t* at;  // of each listed coefficient: element of the warp's inputs, 32 t
  __device__ Smem(unsigned char* raw, int nin, int nout, int warp) {
    off = reinterpret_cast<int64_t*>(raw);
    cnt = reinterpret_cast<int*>(off + 64);
    const int len = list_len(nin, nout);
    at = reinterpret_cast<uint16_t*>(cnt + 64);
    w = reinterpret_cast<T*>(at + len);
    in = w + len + warp * 32 * (nin + (LEFT ? nout : 0));
    out = in + nin * 32;
  }
};

// lists of the coefficients of output o = (v or w) * d + s' over inputs t = (w or v) * d + s, and
// each input's offset from the fibre's first one
template <bool LEFT, typename T>
__device__ void load_w(const Smem<T, LEFT>& s, const double* __restrict__ W, int64_t chi_l, int d, int64_t chi_r,
                       int dl, int dr, int nin, int nout) {
  for (int e = threadIdx.x; e < nin * nout; e += blockDim.x) {
    const int o = e / nin, t = e % nin;
    const int w = LEFT ? t / d : o / d, v = LEFT ? o / d : t / d, si = t % d, so = o % d;
    s.w[e] = T(W[((w * dr + v) * d + si) * d + so]);
  }
  for (int t = threadIdx.x; t < nin; t += blockDim.x)
    s.off[t] = LEFT ? ((t / d) * chi_l * d + t % d) * chi_r : int64_t((t % d) * dr + t / d) * chi_r;
  __syncthreads();
  for (int o = threadIdx.x; o < nout; o += blockDim.x) {
    T* w = s.w + o * nin;
    int n = 0;
    for (int t = 0; t < nin; ++t) {
      const T c = w[t];
      if (nonzero(c)) {
        w[n] = c;  // n <= t
        s.at[o * nin + n++] = uint16_t(32 * t);
      }
    }
    s.cnt[o] = n;
  }
  __syncthreads();
}

// the lane's inputs into its column; true if one of them is Inf or NaN
template <bool LEFT, typename T>
__device__ __forceinline__ bool stage(const Smem<T, LEFT>& s, const T* __restrict__ src, bool live, int nin, int lane) {
  bool bad = false;
  int t = 0;
  for (; t + 10 <= nin; t += 10) {  // D = 5, d = 2: one batch
    T x[10];
#pragma unroll
    for (int i = 0; i < 10; ++i) x[i] = live ? src[s.off[t + i]] : T(0);
#pragma unroll
    for (int i = 0; i < 10; ++i) {
      bad |= not_finite(x[i]);
      s.in[(t + i) * 32 + lane] = x[i];
    }
  }
  for (; t < nin; ++t) {
    const T x = live ? src[s.off[t]] : T(0);
    bad |= not_finite(x);
    s.in[t * 32 + lane] = x;
  }
  return bad;
}

template <bool LEFT, typename T>
__device__ __forceinline__ T combine(const Smem<T, LEFT>& s, int nin, int o, bool dense, int lane) {
  const T* w = s.w + o * nin;
  const uint16_t* at = s.at + o * nin;
  const T* in = s.in + lane;
  const int n = s.cnt[o];
  T acc = T(0);
  if (!dense) {
#pragma unroll 2
    for (int i = 0; i < n; ++i) acc = fma(in[at[i]], w[i], acc);
  } else {
    for (int t = 0, i = 0; t < nin; ++t) {
      const bool listed = i < n && at[i] == 32 * t;
      acc = fma(in[32 * t], listed ? w[i] : T(0), acc);
      i += listed;
    }
  }
  return acc;
}

// idx / n for 0 <= idx, in 32 bits where it fits
__device__ __forceinline__ int64_t quot(int64_t idx, int64_t n) {
  return ((idx | n) >> 32) == 0 ? int64_t(unsigned(idx) / unsigned(n)) : idx / n;
}

// ldp: row pitch of T2 (chi_r * dr, or the padded pitch of a GEMM operand)
template <typename T, typename Out>
__global__ void left_kernel(const T* __restrict__ T1, int64_t sT1, const double* __restrict__ W, int64_t sW, Out out,
                            int64_t sT2, int64_t chi_l, int d, int64_t chi_r, int dl, int dr, int64_t ldp,
                            const int* __restrict__ mask) {
  extern __shared__ __align__(16) unsigned char wc_raw[];
  if (mask && !mask[blockIdx.y]) return;
  const int nin = dl * d, nout = dr * d, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const Smem<T, true> s(wc_raw, nin, nout, warp);
  T1 += blockIdx.y * sT1;
  const int64_t ob = blockIdx.y * sT2;
  load_w<true>(s, W + blockIdx.y * sW, chi_l, d, chi_r, dl, dr, nin, nout);
  const int64_t total = chi_l * chi_r;
  const int qd = 32 / dr, rd = 32 % dr;  // step of (fibre, v) over 32 consecutive outputs
  const int p0 = lane / dr, v0 = lane - p0 * dr;
  const bool in_pairs = out.aligned() && ((ldp | ob) & 1) == 0;
  for (int64_t i0 = (int64_t(blockIdx.x) * nw + warp) * 32; i0 < total; i0 += int64_t(gridDim.x) * nw * 32) {
    const int64_t idx = i0 + lane;
    const int64_t ap = quot(idx, chi_r), c = idx - ap * chi_r;
    const bool dense = __any_sync(0xffffffffu, stage(s, T1 + (ap * d * chi_r + c), idx < total, nin, lane));
    for (int o = 0, v = 0; v < dr; ++v)
      for (int sp = 0; sp < d; ++sp, ++o) s.out[(sp * 32 + lane) * dr + v] = combine(s, nin, o, dense, lane);
    __syncwarp();
    const int np = total - i0 < 32 ? int(total - i0) : 32;
    // the 32 fibres cover c .. c + 31 of row a' and, past the row's end, the start of the next
    const int64_t ap0 = __shfl_sync(0xffffffffu, ap, 0), c0 = __shfl_sync(0xffffffffu, c, 0);
    if (in_pairs && c0 + np <= chi_r && ((c0 * dr) & 1) == 0) {
      const int64_t base = ob + ap0 * d * ldp + c0 * dr;
      for (int sp = 0; sp < d; ++sp) {
        const T* res = s.out + sp * 32 * dr;
        int e = 2 * lane;
        for (; e + 1 < np * dr; e += 64) out.two(base + sp * ldp + e, res + e);
        if (e < np * dr) out.at(base + sp * ldp + e, res[e]);
      }
      __syncwarp();
      continue;
    }
    int p = p0, v = v0;
    for (int e = lane; e < np * dr; e += 32) {
      int64_t pc = c0 + p, pa = ap0;
      if (pc >= chi_r) {
        const int64_t k = quot(pc, chi_r);
        pa += k;
        pc -= k * chi_r;
      }
      const int64_t base = ob + pa * d * ldp + pc * dr + v;
      for (int sp = 0; sp < d; ++sp) out.at(base + sp * ldp, s.out[sp * 32 * dr + e]);
      p += qd;
      v += rd;
      if (v >= dr) {
        v -= dr;
        ++p;
      }
    }
    __syncwarp();  // the outputs are read before the next fibres rewrite them
  }
}

template <typename T>
__global__ void right_kernel(const T* __restrict__ T1, int64_t sT1, const double* __restrict__ W, int64_t sW,
                             T* __restrict__ T2, int64_t sT2, int64_t chi_l, int d, int64_t chi_r, int dl, int dr) {
  extern __shared__ __align__(16) unsigned char wc_raw[];
  const int nin = dr * d, nout = dl * d, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const Smem<T, false> s(wc_raw, nin, nout, warp);
  T1 += blockIdx.y * sT1;
  T2 += blockIdx.y * sT2;
  load_w<false>(s, W + blockIdx.y * sW, chi_l, d, chi_r, dl, dr, nin, nout);
  const int64_t total = chi_l * chi_r;
  for (int64_t i0 = (int64_t(blockIdx.x) * nw + warp) * 32; i0 < total; i0 += int64_t(gridDim.x) * nw * 32) {
    const int64_t idx = i0 + lane;
    const int64_t a = quot(idx, chi_r), c = idx - a * chi_r;
    const bool live = idx < total;
    const bool dense = __any_sync(0xffffffffu, stage(s, T1 + (a * d * dr * chi_r + c), live, nin, lane));
    T* o_base = T2 + a * nout * chi_r + c;
    for (int o = 0; o < nout; ++o) {
      const T r = combine(s, nin, o, dense, lane);
      if (live) o_base[int64_t(o) * chi_r] = r;
    }
  }
}

// warps per CTA (each takes its own fibres) and CTAs
template <typename T, bool LEFT>
int warps_for(int nin, int nout) {
  return sizeof(T) * 32 * (nin + (LEFT ? nout : 0)) <= 8192 ? 4 : 2;
}
inline unsigned ctas_for(int64_t total, int nw) {
  const int64_t b = (total + 32 * nw - 1) / (32 * nw);
  return unsigned(b > 152 * 11 ? 152 * 11 : (b < 1 ? 1 : b));
}

// (internal linkage: a kernel in a header is a translation unit's own, and so is the set of devices that know it)
template <typename T, typename Out>
static int launch_left(const T* T1, int64_t sT1, const double* W, int64_t sW, Out out, int64_t sT2, int64_t chi_l, int64_t d,
                int64_t chi_r, int64_t dl, int64_t dr, int64_t ldp, int batch, const int* mask, cudaStream_t st) {
  const int nin = int(dl * d), nout = int(dr * d), nw = warps_for<T, true>(nin, nout);
  const size_t smem = smem_bytes<T, true>(nin, nout, nw);
  static DeviceSet allowed;
  TNX_CUDA((allow_smem(left_kernel<T, Out>, smem_bytes<T, true>(64, 64, 4), allowed)));  // no MPO takes more
  left_kernel<T, Out><<<dim3(ctas_for(chi_l * chi_r, nw), unsigned(batch)), 32 * nw, smem, st>>>(
      T1, sT1, W, sW, out, sT2, chi_l, int(d), chi_r, int(dl), int(dr), ldp, mask);
  TNX_LAUNCH_CHECK();
  return TNX_OK;
}

template <typename T>
static int launch_right(const T* T1, int64_t sT1, const double* W, int64_t sW, T* T2, int64_t sT2, int64_t chi_l, int64_t d,
                 int64_t chi_r, int64_t dl, int64_t dr, int batch, cudaStream_t st) {
  const int nin = int(dr * d), nout = int(dl * d), nw = warps_for<T, false>(nin, nout);
  const size_t smem = smem_bytes<T, false>(nin, nout, nw);
  static DeviceSet allowed;
  TNX_CUDA((allow_smem(right_kernel<T>, smem_bytes<T, false>(64, 64, 4), allowed)));
  right_kernel<T><<<dim3(ctas_for(chi_l * chi_r, nw), unsigned(batch)), 32 * nw, smem, st>>>(
      T1, sT1, W, sW, T2, sT2, chi_l, int(d), chi_r, int(dl), int(dr));
  TNX_LAUNCH_CHECK();
  return TNX_OK;
}

}  // namespace wc
}  // namespace tnx
