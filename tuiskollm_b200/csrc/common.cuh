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

// max(|.|) of two packed BF16 pairs, NaNs ignored as by fmaxf (`acc` starts at 0).  The signs of the result
// mean nothing; bf16x2_fold gives the bits of the larger magnitude.
__device__ __forceinline__ uint32_t bf16x2_absmax(uint32_t acc, uint32_t w) {
  uint32_t r;
  asm("max.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(acc), "r"(w));
  return r;
}
__device__ __forceinline__ uint32_t bf16x2_fold(uint32_t m) { return max(m & 0x7fffu, (m >> 16) & 0x7fffu); }

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

// 1 / s as the sum hi + lo, hi slightly below it and lo > 0: rcp.approx is within one unit in the last
// place, so three units less is below, and lo = (1 - hi s) hi restores what is missing to 2^-42.  A product
// x hi + x lo, the second part rounded first, is then within 2^-42 of x / s before its one rounding, and keeps
// the sign of a zero x (hence lo > 0).  Two operations per quotient, where a division takes about eight and
// residual steps on a rounded reciprocal three to five; s must leave hi and lo normal (2^-100 .. 2^100).
struct Reciprocal {
  float hi, lo;
};
__device__ __forceinline__ Reciprocal reciprocal_parts(float s) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(s));
  Reciprocal p;
  p.hi = __uint_as_float(__float_as_uint(r) - 3u);
  p.lo = __fmul_rn(__fmaf_rn(-p.hi, s, 1.0f), p.hi);
  return p;
}
__device__ __forceinline__ F32x2 quotient(F32x2 x, F32x2 hi, F32x2 lo) { return fma2(x, hi, mul2(x, lo)); }

// E4M3 row quantiser: scale = amax / 448 (1 for a zero row), code = e4m3_rne_sat(x / scale), both quotients
// rounded as the division rounds them.  amax has 128 significands (it is a BF16 value): for each of them and
// each BF16 x <= amax the two-part products round like the division (all 128 x 128 pairs of significands
// checked), so an ordinary amax takes them; beyond, where exponents run out, the division runs.
__device__ __forceinline__ bool e4m3_amax_is_ordinary(float amax) { return amax >= 0x1p-60f && amax <= 0x1p97f; }
__device__ __forceinline__ float e4m3_scale_ordinary(float amax) {
  // 1 / 448 in two parts, the first three units in the last place below it
  return __fmaf_rn(amax, 0x1.249244p-9f, __fmul_rn(amax, 0x1.49248cp-31f));
}
__device__ __forceinline__ float e4m3_scale(float amax) { return amax == 0.0f ? 1.0f : __fdiv_rn(amax, 448.0f); }
__device__ __forceinline__ uint32_t e4m3_pair_ordinary(F32x2 x, F32x2 hi, F32x2 lo) {
  const float2 q = f32x2_parts(quotient(x, hi, lo));
  return f32x2_to_e4m3x2(q.x, q.y);
}
__device__ __forceinline__ uint32_t e4m3_pair(F32x2 x, float scale) {
  const float2 v = f32x2_parts(x);
  return f32x2_to_e4m3x2(__fdiv_rn(v.x, scale), __fdiv_rn(v.y, scale));
}

// Four pairs of f32 -> eight E2M1 codes (cvt.rn.satfinite.e2m1x2.f32), first value in the lowest nibble.
__device__ __forceinline__ uint32_t f32x8_to_e2m1x8(F32x2 a, F32x2 b, F32x2 c, F32x2 d) {
  const float2 p = f32x2_parts(a), q = f32x2_parts(b), r = f32x2_parts(c), s = f32x2_parts(d);
  uint32_t w;
  asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n\t"
      "mov.b32 %0, {b0, b1, b2, b3};\n\t}"
      : "=r"(w)
      : "f"(p.x), "f"(p.y), "f"(q.x), "f"(q.y), "f"(r.x), "f"(r.y), "f"(s.x), "f"(s.y));
  return w;
}

// Scale code of an NVFP4 block, e4m3_rne_sat((amax * divisor) / 6).  Six times an E4M3 rounding boundary has at
// most 7 significant bits, so a quotient is on a boundary exactly or more than 1.3 half units in the last
// place away from it: the two-part product decides every code as the division does.
__device__ __forceinline__ uint32_t nvfp4_scale_code(float amax, float divisor) {
  constexpr float hi = 0x1.55555p-3f, lo = 0x1.55555p-25f;  // 1 / 6 in two parts, the first below it
  const float t = __fmul_rn(amax, divisor);
  return f32x2_to_e4m3x2(__fmaf_rn(t, hi, __fmul_rn(t, lo)), 0.0f) & 0xffu;
}

// NVFP4 codes of N packed BF16 pairs of one block: code = e2m1_rne_sat((x * divisor) / s), signed zeros
// when s == 0; two codes a byte, low nibble first.  s is a decoded E4M3 scale (4 significant bits) and an
// E2M1 rounding boundary has 3, so a quotient is on a boundary exactly or more than 1.007 half units in
// the last place away from it: the two-part product decides every code as the division does.
template <int N>
__device__ __forceinline__ void nvfp4_codes(const F32x2 (&x)[N], float divisor, float s, uint32_t (&packed)[N / 4]) {
  if (s == 0.0f) {
#pragma unroll
    for (int j = 0; j < N / 4; ++j) {
      packed[j] = 0u;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 v = f32x2_parts(x[4 * j + i]);
        const uint32_t byte = ((__float_as_uint(v.x) >> 28) & 0x08u) | ((__float_as_uint(v.y) >> 24) & 0x80u);
        packed[j] |= byte << (8 * i);
      }
    }
    return;
  }
  const Reciprocal r = reciprocal_parts(s);
  const F32x2 div = f32x2_splat(divisor), hi = f32x2_splat(r.hi), lo = f32x2_splat(r.lo);
#pragma unroll
  for (int j = 0; j < N / 4; ++j) {
    F32x2 q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) q[i] = quotient(mul2(x[4 * j + i], div), hi, lo);
    packed[j] = f32x8_to_e2m1x8(q[0], q[1], q[2], q[3]);
  }
}

// The quotient of one value that its code is rounded from, as nvfp4_codes forms it.
__device__ __forceinline__ float nvfp4_quotient(float x, float divisor, float s) {
  const Reciprocal r = reciprocal_parts(s);
  const float t = __fmul_rn(x, divisor);
  return s == 0.0f ? copysignf(0.0f, x) : __fmaf_rn(t, r.hi, __fmul_rn(t, r.lo));
}

// NVFP4 form of 16 consecutive BF16 values (8 packed pairs, low half first):
//   scale = e4m3_rne_sat((amax * divisor) / 6),  code = e2m1_rne_sat((x * divisor) / scale),
// signed zeros when the scale underflows to 0.  Codes low nibble first.
__device__ __forceinline__ uint2 nvfp4_quantize_block(const uint32_t (&w)[8], float divisor, uint32_t* scale_code) {
  uint32_t m = 0u;
  F32x2 x[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    m = bf16x2_absmax(m, w[j]);
    x[j] = bf16x2_to_f32x2(w[j]);
  }
  const uint32_t sc = nvfp4_scale_code(__uint_as_float(bf16x2_fold(m) << 16), divisor);
  *scale_code = sc;
  uint32_t packed[2];
  nvfp4_codes(x, divisor, e4m3_to_f32(sc), packed);
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

}  // namespace tk100
