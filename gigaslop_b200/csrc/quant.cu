// Per-token (per-row) absmax quantisers: fp16/fp32 [M,K] -> int8 or E4M3 [M,K]
// plus one fp32 dequantisation scale per row.  HBM-bound: each row is read once
// with 16/32-byte vector loads, held in registers across the warp-shuffle max
// reduction, and written once with 8-byte stores.  One warp owns one row.
//
// The arithmetic order is part of the contract (results are bit-exact against the
// CPU reference): INT8 uses qs = (1/amax)*127, q = rne(x*qs), scale = 1/qs; FP8 has the kernel formulation (x * (448/amax)) and the torch formulation
// (x / (amax/448)).
#include <cuda_fp8.h>

#include "capi_internal.h"
#include "ptx.cuh"

namespace gsb {

constexpr int QUANT_WARPS = 8;

template <typename Tin>
__device__ __forceinline__ void load8(const Tin* p, float (&v)[8]);

template <>
__device__ __forceinline__ void load8<__half>(const __half* p, float (&v)[8]) {
  const uint4 raw = __ldcs(reinterpret_cast<const uint4*>(p));
  const __half2* h = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __half22float2(h[i]);
    v[2 * i] = f.x; v[2 * i + 1] = f.y;
  }
}
template <>
__device__ __forceinline__ void load8<float>(const float* p, float (&v)[8]) {
  const float4 a = __ldcs(reinterpret_cast<const float4*>(p));
  const float4 b = __ldcs(reinterpret_cast<const float4*>(p + 4));
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

__device__ __forceinline__ float warp_max(float m) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
  return m;
}

// Two int32 -> two saturated int8 in the low half of the result, the low half of `upper` above them:
// result = upper[15:0] << 16 | sat8(hi) << 8 | sat8(lo).
__device__ __forceinline__ uint32_t pack_sat_s8(int hi, int lo, uint32_t upper) {
  uint32_t d;
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(hi), "r"(lo), "r"(upper));
  return d;
}
// q = clamp(rne(x * qs), -127, 127) for four values, packed little-endian.  |x| <= amax and qs = fl(fl(1/amax)*127)
// bound |x*qs| by 127.0001, so the rounded value never leaves [-127, 127]; the pack saturates all the same.
__device__ __forceinline__ uint32_t pack4_i8(float x0, float x1, float x2, float x3, float qs) {
  const float2 q2 = make_float2(qs, qs);
  const float2 a = __fmul2_rn(make_float2(x0, x1), q2), b = __fmul2_rn(make_float2(x2, x3), q2);
  const uint32_t hi = pack_sat_s8(__float2int_rn(b.y), __float2int_rn(b.x), 0u);     // round half to even
  return pack_sat_s8(__float2int_rn(a.y), __float2int_rn(a.x), hi);
}

__device__ __forceinline__ uint2 pack_i8(const float (&v)[8], float qs) {
  uint2 o;
  o.x = pack4_i8(v[0], v[1], v[2], v[3], qs);
  o.y = pack4_i8(v[4], v[5], v[6], v[7], qs);
  return o;
}

// FP8: mode 0 multiplies by inv = 448/amax; mode 1 divides by scale = amax/448 and clamps.
template <int MODE>
__device__ __forceinline__ float fp8_prescale(float x, float f) {
  if constexpr (MODE == 0) return __fmul_rn(x, f);
  else return fminf(fmaxf(__fdiv_rn(x, f), -448.f), 448.f);
}
template <int MODE>
__device__ __forceinline__ uint2 pack_e4m3(const float (&v)[8], float f) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 pr = make_float2(fp8_prescale<MODE>(v[2 * i], f), fp8_prescale<MODE>(v[2 * i + 1], f));
    w[i] = __nv_cvt_float2_to_fp8x2(pr, __NV_SATFINITE, __NV_E4M3);    // rn, saturate to +-448
  }
  uint2 o;
  o.x = w[0] | (w[1] << 16);
  o.y = w[2] | (w[3] << 16);
  return o;
}

// e4m3( clamp(x / s) ) for a row whose values are all finite, without a division per element: with r = 1 / s correctly
// rounded and q within one ulp of x / s, q + (x - s q) r rounds to the correctly rounded quotient (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1), 1990).  x r itself
// can be 1.5 ulp off, so in general the step is made twice.  For fp16 rows once is enough (HALF): the value that the first step
// rounds is within 2^-46 of x / s, so its fp32 rounding, and with it the E4M3 byte, can only be wrong where x / s lies that close to
// m (1 + 2^-24) or m (1 - 2^-25 or 2^-24), m halfway between two E4M3 values, i.e. up to five significant bits.  In integers, X an
// 11-bit, S a 24-bit significand and m = 16 .. 31: |X 2^k - S (m 2^20 +- 1)| <= 8 needs S = c 2^20 + e, |e| <= 8, and e m = +-c, which
// leaves m = c = 16, e = -1; but s = fl(amax / 448) of an fp16 amax is never the fp32 number below a power of two (amax / 7 would
// have to be within 2^-24 of one without being it).  The residual is inexact only where |x| < 2^-100, and x / s is then far
// below half of the smallest E4M3 value (s >= 2^-49) whatever its last bit; |x| <= 448 s, so the saturating conversion is
// the clamp.  Everything is carried with the opposite sign, so that a zero keeps its own: the additions round +0 + -0 to
// +0, and the sign bits are flipped in the packed bytes.
// With a division per element (about ten instructions) the kernel was issue-bound: M = 131072, K = 1024 took 87.5 us,
// 4.6 TB/s, and M = 9001, K = 2048 14.0 us; with the step made twice 64.8 us and 9.9, once 60.0 us (6.7 TB/s) and 8.8.  K = 512: M =
// 20001 7.3 us twice, 6.5 once, M = 65536 19.0 and 16.5.
template <bool HALF>
__device__ __forceinline__ uint2 pack_e4m3_quot(const float (&v)[8], float s, float neg_r) {
  const float2 s2 = make_float2(s, s), n2 = make_float2(neg_r, neg_r);
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 x = make_float2(v[2 * i], v[2 * i + 1]);
    float2 q = __fmul2_rn(x, n2);                        // -x / s
    q = __ffma2_rn(__ffma2_rn(q, s2, x), n2, q);
    if constexpr (!HALF) q = __ffma2_rn(__ffma2_rn(q, s2, x), n2, q);
    w[i] = __nv_cvt_float2_to_fp8x2(q, __NV_SATFINITE, __NV_E4M3);
  }
  return make_uint2((w[0] | (w[1] << 16)) ^ 0x80808080u, (w[2] | (w[3] << 16)) ^ 0x80808080u);
}

// This warp's row.  The rows are walked from the last to the first: the GEMMs walk theirs upwards, so a quantiser starts
// with the rows its producer wrote last and leaves the rows its consumer reads first written last.  Where a tensor is
// larger than L2 (126 MB) that is what is found there.  The input is read with the streaming hint, so that it does not push
// the output out.  Feed-forward passes of 65536 rows, a few back to back at the full clock: INT8 240.7 -> 234.2 us (walked
// backwards) -> 229.1 (streaming hint), MXFP8 285 -> 281 -> 276.  (In runs of a second the power cap takes the clock from 1965
// to about 1510 MHz and the INT8 pass to 268 us.)
__device__ __forceinline__ long long quant_row() {
  return (long long)(gridDim.x - 1 - blockIdx.x) * QUANT_WARPS + (threadIdx.x >> 5);
}

// FMT: 0 = int8, 1 = e4m3 kernel formulation, 2 = e4m3 torch formulation.
// NV > 0: the row (<= NV*256 elements) is cached in registers.  NV == 0: any K, second pass re-reads.
template <typename Tin, int FMT, int NV>
__global__ void __launch_bounds__(QUANT_WARPS * 32)
ptq_kernel(const Tin* __restrict__ x, long long ldx, uint8_t* __restrict__ q, long long ldq,
           float* __restrict__ scale, long long M, int K) {
  const int lane = threadIdx.x & 31;
  const long long row = quant_row();
  pdl_wait();
  pdl_trigger();
  if (row >= M) return;
  const Tin* xr = x + row * ldx;
  uint8_t* qr = q + row * ldq;
  const int nvec = K >> 3;

  float vals[NV > 0 ? NV : 1][8];
  float amax = 0.f;
  bool bad = false;                      // FMT 2: the row holds a NaN (or, below, an infinity)
  constexpr bool HALF_CACHED = NV > 0 && sizeof(Tin) == 2;
  uint4 raw[HALF_CACHED ? NV : 1];       // fp16 rows are held as loaded: 8 halves per 16-byte vector
  if constexpr (HALF_CACHED) {
    // row maximum with packed half2 max / abs (exact: it is a maximum of the very same fp16 values)
    __half2 m2 = __float2half2_rn(0.f), any2 = m2;       // any2 keeps a NaN that the maximum skips
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = lane + 32 * i;
      raw[i] = make_uint4(0u, 0u, 0u, 0u);
      if (v < nvec) raw[i] = __ldcs(reinterpret_cast<const uint4*>(xr + v * 8));
      const __half2* h = reinterpret_cast<const __half2*>(&raw[i]);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        m2 = __hmax2(m2, __habs2(h[k]));
        if constexpr (FMT == 2) any2 = __hmax2_nan(any2, __habs2(h[k]));
      }
    }
    amax = fmaxf(__low2float(m2), __high2float(m2));
    if constexpr (FMT == 2) bad = __hisnan(__low2half(any2)) || __hisnan(__high2half(any2));
  } else if constexpr (NV > 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = lane + 32 * i;
      if (v < nvec) {
        load8<Tin>(xr + v * 8, vals[i]);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          amax = fmaxf(amax, fabsf(vals[i][j]));
          if constexpr (FMT == 2) bad |= vals[i][j] != vals[i][j];
        }
      }
    }
  } else {
    for (int v = lane; v < nvec; v += 32) {
      load8<Tin>(xr + v * 8, vals[0]);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        amax = fmaxf(amax, fabsf(vals[0][j]));
        if constexpr (FMT == 2) bad |= vals[0][j] != vals[0][j];
      }
    }
  }
  amax = warp_max(amax);

  float f;   // factor applied to the elements
  float s;   // dequantisation scale written out
  if constexpr (FMT == 0) {
    amax = fmaxf(amax, 1e-8f);
    // the reference computes `127 / amax` with a Python scalar numerator, which PyTorch evaluates as
    // reciprocal(amax) * 127 (two roundings) -- reproduced here so every int8 value matches
    f = __fmul_rn(__frcp_rn(amax), 127.0f);
    s = __frcp_rn(f);
  } else {
    amax = fmaxf(amax, 1e-12f);
    s = __fdiv_rn(amax, 448.0f);
    f = (FMT == 1) ? __fdiv_rn(448.0f, amax) : s;
  }
  if (lane == 0) scale[row] = s;
  [[maybe_unused]] float neg_r = 0.f;
  if constexpr (FMT == 2) {
    bad = __any_sync(0xffffffffu, bad) || !(amax <= 3.402823466e38f);
    neg_r = -__frcp_rn(s);
  }

  auto emit = [&](int v, const float (&vv)[8]) {
    uint2 o;
    if constexpr (FMT == 0) o = pack_i8(vv, f);
    else if constexpr (FMT == 1) o = pack_e4m3<0>(vv, f);
    else if (bad) o = pack_e4m3<1>(vv, f);       // warp-uniform: only rows with a NaN or an infinity divide
    else o = pack_e4m3_quot<sizeof(Tin) == 2>(vv, s, neg_r);
    *reinterpret_cast<uint2*>(qr + v * 8) = o;
  };
  if constexpr (HALF_CACHED) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = lane + 32 * i;
      if (v < nvec) {
        const __half2* h = reinterpret_cast<const __half2*>(&raw[i]);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 f2 = __half22float2(h[k]);
          vals[0][2 * k] = f2.x; vals[0][2 * k + 1] = f2.y;
        }
        emit(v, vals[0]);
      }
    }
  } else if constexpr (NV > 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = lane + 32 * i;
      if (v < nvec) emit(v, vals[i]);
    }
  } else {
    for (int v = lane; v < nvec; v += 32) {
      load8<Tin>(xr + v * 8, vals[0]);
      emit(v, vals[0]);
    }
  }
}

template <typename Tin, int FMT>
static cudaError_t launch_fmt(const void* x, long long ldx, void* q, long long ldq, float* scale, long long M, int K,
                              cudaStream_t st) {
  const unsigned blocks = (unsigned)((M + QUANT_WARPS - 1) / QUANT_WARPS);
  const Tin* xp = static_cast<const Tin*>(x);
  uint8_t* qp = static_cast<uint8_t*>(q);
  cudaError_t e;
  if (K <= 512) e = launch_dependent(ptq_kernel<Tin, FMT, 2>, blocks, QUANT_WARPS * 32, 0, st, xp, ldx, qp, ldq, scale, M, K);
  else if (K <= 1024) e = launch_dependent(ptq_kernel<Tin, FMT, 4>, blocks, QUANT_WARPS * 32, 0, st, xp, ldx, qp, ldq, scale, M, K);
  else if (K <= 2048) e = launch_dependent(ptq_kernel<Tin, FMT, 8>, blocks, QUANT_WARPS * 32, 0, st, xp, ldx, qp, ldq, scale, M, K);
  else e = launch_dependent(ptq_kernel<Tin, FMT, 0>, blocks, QUANT_WARPS * 32, 0, st, xp, ldx, qp, ldq, scale, M, K);
  return e;
}

// ---- MXFP8 activation quantiser: E4M3 elements + one E8M0 scale per 32 consecutive elements of a row -------
// scale byte = clamp(biased_exponent(block max) - 8, 0, 254), elements = e4m3_rn_satfinite(x * 2^(127-byte)).
// A lane owns 8 consecutive elements, so a 32-element block lives in 4 neighbouring lanes (two xor-shuffles).  HBM-bound:
// all NV vectors of a lane are loaded before the first is used (with one load in flight per lane and 256-element step the
// kernel waited for memory: M = 65536, K = 512 22.6 us and K = 2048 84 us; now 17.7 and 62.4 us, 6.5 TB/s), and the block maximum of fp16 rows is taken
// with packed half2 instructions (exact, like the per-token kernel's).
template <typename Tin, int NV>
__global__ void __launch_bounds__(QUANT_WARPS * 32)
ptq_mx_kernel(const Tin* __restrict__ x, long long ldx, uint8_t* __restrict__ q, long long ldq,
              uint8_t* __restrict__ scales, long long lds, long long M, int K) {
  const int lane = threadIdx.x & 31;
  const long long row = quant_row();
  pdl_wait();
  pdl_trigger();
  if (row >= M) return;
  const Tin* xr = x + row * ldx;
  constexpr bool HALF = sizeof(Tin) == 2;
  constexpr int WORDS = HALF ? 1 : 2;              // 16-byte words of 8 elements
  const int nvec = K >> 3;                         // K % 32 == 0 -> nvec % 4 == 0: the 4 lanes of a block agree on `v < nvec`
  for (int v0 = 0; v0 < nvec; v0 += 32 * NV) {
    uint4 raw[NV][WORDS];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = v0 + 32 * i + lane;
#pragma unroll
      for (int w = 0; w < WORDS; ++w) {
        raw[i][w] = make_uint4(0u, 0u, 0u, 0u);
        if (v < nvec) raw[i][w] = __ldcs(reinterpret_cast<const uint4*>(xr + v * 8) + w);
      }
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = v0 + 32 * i + lane;
      float vals[8];
      float amax;
      if constexpr (HALF) {
        const __half2* h = reinterpret_cast<const __half2*>(&raw[i][0]);
        const __half2 m2 = __hmax2(__hmax2(__habs2(h[0]), __habs2(h[1])), __hmax2(__habs2(h[2]), __habs2(h[3])));
        amax = fmaxf(fmaxf(__low2float(m2), __high2float(m2)), 0.f);        // (a block of NaNs counts as zero)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 f2 = __half22float2(h[k]);
          vals[2 * k] = f2.x; vals[2 * k + 1] = f2.y;
        }
      } else {
        amax = 0.f;
#pragma unroll
        for (int w = 0; w < WORDS; ++w) {
          const float* f = reinterpret_cast<const float*>(&raw[i][w]);
#pragma unroll
          for (int k = 0; k < 4; ++k) { vals[4 * w + k] = f[k]; amax = fmaxf(amax, fabsf(f[k])); }
        }
      }
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
      if (v < nvec) {
        int eb = (int)((__float_as_uint(amax) >> 23) & 0xffu) - 8;
        eb = max(0, min(254, eb));
        const float inv = __uint_as_float((uint32_t)(254 - eb) << 23);
        *reinterpret_cast<uint2*>(q + row * ldq + v * 8) = pack_e4m3<0>(vals, inv);
        if ((lane & 3) == 0) scales[row * lds + (v >> 2)] = (uint8_t)eb;
      }
    }
  }
}

template <typename Tin>
static cudaError_t launch_mx_rows(const void* x, long long ldx, uint8_t* q, long long ldq, uint8_t* scales, long long lds, long long M,
                           int K, cudaStream_t st) {
  const unsigned blocks = (unsigned)((M + QUANT_WARPS - 1) / QUANT_WARPS);
  const Tin* xp = static_cast<const Tin*>(x);
  if (K <= 256) return launch_dependent(ptq_mx_kernel<Tin, 1>, blocks, QUANT_WARPS * 32, 0, st, xp, ldx, q, ldq, scales, lds, M, K);
  if (K <= 512) return launch_dependent(ptq_mx_kernel<Tin, 2>, blocks, QUANT_WARPS * 32, 0, st, xp, ldx, q, ldq, scales, lds, M, K);
  return launch_dependent(ptq_mx_kernel<Tin, 4>, blocks, QUANT_WARPS * 32, 0, st, xp, ldx, q, ldq, scales, lds, M, K);
}

int32_t launch_ptq_mx(const void* x, int x_dtype, long long ldx, uint8_t* q, long long ldq, uint8_t* scales,
                      long long lds, long long M, int K, cudaStream_t st) {
  if (M == 0) return GSB200_OK;
  if (!x || !q || !scales || M < 0 || K <= 0 || K % 32 != 0) return GSB200_ERR_BAD_ARG;
  if (ldx < K || ldq < K || ldq % 8 != 0 || lds < K / 32) return GSB200_ERR_BAD_ARG;
  if (x_dtype != GSB200_F16 && x_dtype != GSB200_F32) return GSB200_ERR_BAD_ARG;
  const int esz = x_dtype == GSB200_F16 ? 2 : 4;
  if ((ldx * esz) % 16 != 0 || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(q) & 7))
    return GSB200_ERR_BAD_ARG;
  if ((M + QUANT_WARPS - 1) / QUANT_WARPS > 0x7fffffffll) return GSB200_ERR_BAD_ARG;
  const cudaError_t e = x_dtype == GSB200_F16 ? launch_mx_rows<__half>(x, ldx, q, ldq, scales, lds, M, K, st)
                                              : launch_mx_rows<float>(x, ldx, q, ldq, scales, lds, M, K, st);
  return cuda_status(e, "ptq_mx launch");
}

int32_t launch_ptq(const void* x, int x_dtype, long long ldx, void* q, long long ldq, float* scale, long long M, int K,
                   int fmt, cudaStream_t st) {
  if (M == 0) return GSB200_OK;
  if (!x || !q || !scale || M < 0 || K <= 0) return GSB200_ERR_BAD_ARG;
  if (K % 8 != 0 || ldx < K || ldq < K || ldq % 8 != 0) return GSB200_ERR_BAD_ARG;
  const int esz = x_dtype == GSB200_F16 ? 2 : 4;
  if (x_dtype != GSB200_F16 && x_dtype != GSB200_F32) return GSB200_ERR_BAD_ARG;
  if ((ldx * esz) % 16 != 0 || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(q) & 7))
    return GSB200_ERR_BAD_ARG;
  if ((M + QUANT_WARPS - 1) / QUANT_WARPS > 0x7fffffffll) return GSB200_ERR_BAD_ARG;
  cudaError_t e;
  if (x_dtype == GSB200_F16) {
    if (fmt == 0) e = launch_fmt<__half, 0>(x, ldx, q, ldq, scale, M, K, st);
    else if (fmt == 1) e = launch_fmt<__half, 1>(x, ldx, q, ldq, scale, M, K, st);
    else if (fmt == 2) e = launch_fmt<__half, 2>(x, ldx, q, ldq, scale, M, K, st);
    else return GSB200_ERR_BAD_ARG;
  } else {
    if (fmt == 0) e = launch_fmt<float, 0>(x, ldx, q, ldq, scale, M, K, st);
    else if (fmt == 1) e = launch_fmt<float, 1>(x, ldx, q, ldq, scale, M, K, st);
    else if (fmt == 2) e = launch_fmt<float, 2>(x, ldx, q, ldq, scale, M, K, st);
    else return GSB200_ERR_BAD_ARG;
  }
  return cuda_status(e, "ptq launch");
}

}  // namespace gsb
