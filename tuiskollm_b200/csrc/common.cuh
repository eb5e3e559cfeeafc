// Shared device helpers: BF16 / E4M3 / E2M1 conversions with the exact rounding the
// qualification oracles pin, and small block-wide reductions with a fixed order.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp4.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace tk100 {

__device__ __forceinline__ float bf16_bits_to_f32(uint32_t bits16) {
  return __uint_as_float(bits16 << 16);
}

// Low half = element 2j, high half = element 2j+1 of a packed BF16 pair.
__device__ __forceinline__ float bf16x2_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16x2_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// Round-to-nearest-even f32 -> BF16 bits (cvt.rn.bf16.f32).
__device__ __forceinline__ uint32_t f32_to_bf16_bits(float v) {
  return static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(v)));
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  return f32_to_bf16_bits(lo) | (f32_to_bf16_bits(hi) << 16);
}

// Two f32 -> two E4M3FN codes, round-to-nearest-even, saturating to +-448
// (cvt.rn.satfinite.e4m3x2.f32); `lo` lands in the low byte.
__device__ __forceinline__ uint32_t f32x2_to_e4m3x2(float lo, float hi) {
  return static_cast<uint32_t>(
      __nv_cvt_float2_to_fp8x2(make_float2(lo, hi), __NV_SATFINITE, __NV_E4M3));
}

// One E4M3FN code -> f32 (exact).
__device__ __forceinline__ float e4m3_to_f32(uint32_t code) {
  __half_raw h = __nv_cvt_fp8_to_halfraw(static_cast<__nv_fp8_storage_t>(code), __NV_E4M3);
  return __half2float(__half(h));
}

// Two f32 -> two E2M1 codes in one byte, nearest-even, saturating to +-6
// (cvt.rn.satfinite.e2m1x2.f32); `lo` lands in the low nibble.
__device__ __forceinline__ uint32_t f32x2_to_e2m1x2(float lo, float hi) {
  return static_cast<uint32_t>(
      __nv_cvt_float2_to_fp4x2(make_float2(lo, hi), __NV_E2M1, cudaRoundNearest));
}

// silu(v) in the sign-stable form of the reference's NVFP4 route
// (tuisko-kernels-sm89/src/nvfp4/swiglu.rs:142-155), ex2.approx for the exponential.
__device__ __forceinline__ float silu_stable(float v) {
  const float e = -fabsf(v) * 1.4426950408889634f;
  float ex;  // .ftz: 2^e below the normal range reads as 0, as the e < -126 cut-off did
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(ex) : "f"(e));
  return __fdividef(v >= 0.0f ? v : v * ex, 1.0f + ex);
}

// SiLU in the dense-FP8 path's form, v / (1 + ex2(-v * log2 e)) (tuisko-kernels-sm120
// device/fp8_swiglu.rs:13-15).
__device__ __forceinline__ float silu_fp8_path(float v) {
  float ex;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(ex) : "f"(-v * 1.4426950408889634f));
  return __fdividef(v, 1.0f + ex);
}

// t / s for a NVFP4 block: s is a decoded E4M3 scale (4 significant bits), inv = __frcp_rn(s).  One
// residual step on the reciprocal's product (P. Markstein, "Computation of elementary functions on the
// IBM RISC System/6000 processor", IBM J. Res. Dev. 34 (1990), theorem on the corrected quotient)
// rounds like the division wherever an E2M1 code depends on it; quotients below the first rounding
// boundary (signed zeros among them), past the saturation point, infinities and NaNs keep the product.
__device__ __forceinline__ float nvfp4_quotient(float t, float s, float inv) {
  const float q = __fmul_rn(t, inv);
  const float corrected = __fmaf_rn(__fmaf_rn(-q, s, t), inv, q);
  return (fabsf(q) > 0.125f && fabsf(q) < 8.0f) ? corrected : q;
}

// NVFP4 form of 16 consecutive BF16 values (8 packed pairs, low half first):
//   scale = e4m3_rne_sat((amax * divisor) / 6),  code = e2m1_rne_sat((x * divisor) / scale),
// signed zeros when the scale underflows to 0.  Codes low nibble first.
__device__ __forceinline__ uint2 nvfp4_quantize_block(const uint32_t (&w)[8], float divisor, uint32_t* scale_code) {
  float amax = 0.0f;
#pragma unroll
  for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fmaxf(fabsf(bf16x2_lo(w[j])), fabsf(bf16x2_hi(w[j]))));
  const uint32_t sc = f32x2_to_e4m3x2(__fdiv_rn(__fmul_rn(amax, divisor), 6.0f), 0.0f) & 0xffu;
  *scale_code = sc;
  const float s = e4m3_to_f32(sc);
  uint32_t packed[2] = {0u, 0u};
  if (s == 0.0f) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t byte = ((w[j] & 0x8000u) ? 0x08u : 0u) | ((w[j] & 0x80000000u) ? 0x80u : 0u);
      packed[j >> 2] |= byte << (8 * (j & 3));
    }
  } else {
    const float inv = __frcp_rn(s);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t byte = f32x2_to_e2m1x2(nvfp4_quotient(__fmul_rn(bf16x2_lo(w[j]), divisor), s, inv),
                                            nvfp4_quotient(__fmul_rn(bf16x2_hi(w[j]), divisor), s, inv)) & 0xffu;
      packed[j >> 2] |= byte << (8 * (j & 3));
    }
  }
  return make_uint2(packed[0], packed[1]);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Block-wide sum / max with a fixed evaluation order (bit-reproducible across
// launches): butterfly inside each warp, then every thread folds the per-warp
// values in warp order.  `scratch` holds one float per warp.
template <bool IS_MAX>
__device__ __forceinline__ float block_reduce(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int warps = (blockDim.x + 31) >> 5;
  v = IS_MAX ? warp_max(v) : warp_sum(v);
  __syncthreads();  // scratch may still be read from a previous reduction
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float r = scratch[0];
  for (int i = 1; i < warps; ++i) r = IS_MAX ? fmaxf(r, scratch[i]) : r + scratch[i];
  return r;
}

}  // namespace tk100
