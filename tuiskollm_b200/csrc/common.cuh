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
  uint32_t w;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w) : "f"(hi), "f"(lo));
  return w;
}

// Two fp32 values in a 64-bit register; each operation is the IEEE one on both halves, in one issue slot.
using F32x2 = unsigned long long;
__device__ __forceinline__ F32x2 f32x2(float lo, float hi) {
  F32x2 v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ F32x2 f32x2_splat(float v) { return f32x2(v, v); }
__device__ __forceinline__ F32x2 bf16x2_to_f32x2(uint32_t w) { return f32x2(bf16x2_lo(w), bf16x2_hi(w)); }
__device__ __forceinline__ float2 f32x2_parts(F32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ F32x2 add2(F32x2 a, F32x2 b) {
  F32x2 v;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
  return v;
}
__device__ __forceinline__ F32x2 mul2(F32x2 a, F32x2 b) {
  F32x2 v;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
  return v;
}
__device__ __forceinline__ F32x2 fma2(F32x2 a, F32x2 b, F32x2 c) {
  F32x2 v;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
  return v;
}
__device__ __forceinline__ uint32_t f32x2_to_bf16x2(F32x2 v) {
  const float2 f = f32x2_parts(v);
  return pack_bf16x2(f.x, f.y);
}

// max(|.|) of two packed BF16 pairs, NaNs ignored as by fmaxf (`acc` starts at 0).
__device__ __forceinline__ uint32_t bf16x2_absmax(uint32_t acc, uint32_t w) {
  uint32_t r;
  asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(acc), "r"(w & 0x7fff7fffu));
  return r;
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

// x / s by a residual step on the product with the correctly rounded reciprocal (P. Markstein, "Computation
// of elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34 (1990)).  Operands
// come negated: `negative` = -x, ninv = -__frcp_rn(s); that keeps the sign of a zero quotient, which the
// residual of the plain form (0 - 0) would lose.  One step lands within one unit in the last place and
// exactly on every quotient that fp32 holds; a second one rounds like the division.
__device__ __forceinline__ F32x2 quotient_step(F32x2 q, F32x2 negative, F32x2 s, F32x2 ninv) {
  return fma2(fma2(q, s, negative), ninv, q);
}

// E4M3 codes of a packed BF16 pair divided by `scale` (e4m3_rn_satfinite of the IEEE quotient).  Two
// residual steps; they need a scale whose residuals stay in the normal range (e4m3_scale_is_ordinary).
__device__ __forceinline__ bool e4m3_scale_is_ordinary(float scale) { return scale >= 0x1p-80f && scale <= 0x1p120f; }
__device__ __forceinline__ uint32_t e4m3_pair_ordinary(uint32_t w, F32x2 scale, F32x2 ninv) {
  const F32x2 n = bf16x2_to_f32x2(w ^ 0x80008000u);
  const float2 q = f32x2_parts(quotient_step(quotient_step(mul2(n, ninv), n, scale, ninv), n, scale, ninv));
  return f32x2_to_e4m3x2(q.x, q.y);
}
__device__ __forceinline__ uint32_t e4m3_pair(uint32_t w, float scale) {
  return f32x2_to_e4m3x2(__fdiv_rn(bf16x2_lo(w), scale), __fdiv_rn(bf16x2_hi(w), scale));
}

// NVFP4 codes of N packed BF16 pairs of one block: code = e2m1_rne_sat((x * divisor) / s), signed zeros
// when s == 0; two codes a byte, low nibble first.  s is a decoded E4M3 scale (4 significant bits) and an
// E2M1 rounding boundary has 3, so a quotient is on a boundary exactly or more than 1.007 half units in
// the last place away from it: one residual step decides every code as the division does.  An infinite
// product keeps the division (its residual is NaN).
template <int N>
__device__ __forceinline__ void nvfp4_codes(const uint32_t (&w)[N], float block_max, float divisor, float s,
                                            uint32_t (&packed)[N / 4]) {
#pragma unroll
  for (int j = 0; j < N / 4; ++j) packed[j] = 0u;
  if (s == 0.0f) {
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const uint32_t byte = ((w[j] & 0x8000u) ? 0x08u : 0u) | ((w[j] & 0x80000000u) ? 0x80u : 0u);
      packed[j >> 2] |= byte << (8 * (j & 3));
    }
  } else if (__fmul_rn(block_max, divisor) <= 3.0e38f) {
    const F32x2 ndiv = f32x2_splat(-divisor), ninv = f32x2_splat(-__frcp_rn(s)), s2 = f32x2_splat(s);
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const F32x2 n = mul2(bf16x2_to_f32x2(w[j]), ndiv);
      const float2 q = f32x2_parts(quotient_step(mul2(n, ninv), n, s2, ninv));
      packed[j >> 2] |= (f32x2_to_e2m1x2(q.x, q.y) & 0xffu) << (8 * (j & 3));
    }
  } else {
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const uint32_t byte = f32x2_to_e2m1x2(__fdiv_rn(__fmul_rn(bf16x2_lo(w[j]), divisor), s),
                                            __fdiv_rn(__fmul_rn(bf16x2_hi(w[j]), divisor), s));
      packed[j >> 2] |= (byte & 0xffu) << (8 * (j & 3));
    }
  }
}

// NVFP4 form of 16 consecutive BF16 values (8 packed pairs, low half first):
//   scale = e4m3_rne_sat((amax * divisor) / 6),  code = e2m1_rne_sat((x * divisor) / scale),
// signed zeros when the scale underflows to 0.  Codes low nibble first.
__device__ __forceinline__ uint2 nvfp4_quantize_block(const uint32_t (&w)[8], float divisor, uint32_t* scale_code) {
  uint32_t m = 0u;
#pragma unroll
  for (int j = 0; j < 8; ++j) m = bf16x2_absmax(m, w[j]);
  const float amax = fmaxf(bf16x2_lo(m), bf16x2_hi(m));
  const uint32_t sc = f32x2_to_e4m3x2(__fdiv_rn(__fmul_rn(amax, divisor), 6.0f), 0.0f) & 0xffu;
  *scale_code = sc;
  uint32_t packed[2];
  nvfp4_codes(w, amax, divisor, e4m3_to_f32(sc), packed);
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
