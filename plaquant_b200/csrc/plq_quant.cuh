// Device arithmetic of the NVFP4 / MXFP8 quantiser.
//
// Every function reproduces, bit for bit on bf16-valued inputs, what the reference's float32
// fake quantiser computes (promix/quantize/quant_utils.py:660-751), but without its
// 127-entry table scans and IEEE divisions:
//   * NVFP4 scale:  smallest E4M3 value s with s >= fl(max/6).  For a bf16 max this is the
//     smallest s with 6*s >= max (6*s is exact in float32 and a bf16 value can never sit
//     within float32 rounding distance of 6*s without being equal to it), so a hardware
//     round-to-nearest conversion plus one exact comparison finds it.
//   * NVFP4 element: E2M1 code of fl(x/s), from one multiplication x*r rounded toward zero with
//     r = fl(1/s) (the hardware approximation equals it for all 126 scales).  x/s is either exactly a rounding midpoint m or at least 2^-9 (relative) away from
//     every midpoint, so only x == m*s is delicate: fl(1/s) never lies below 1/s (true for the eight
//     significands an E4M3 value can have), the product is m(1 + e) with 0 <= e < one ulp, and rounding
//     toward zero returns m itself; the hardware RNE conversion then breaks the tie like the
//     reference's correctly rounded quotient.  (Before: the quotient refined by two more multiply-adds;
//     together with unit indexes advanced instead of divided, [8192, 14336] rotation + pack went from
//     80.4 to 70.1 us.)
//   * MXFP8 scale: 2^e with the smallest e such that 448*2^e >= max, read off the bf16
//     exponent and mantissa; element: x * 2^-e is exact, then hardware RNE to E4M3.
//   * sign of zero: the reference multiplies the rounded magnitude by sign(x/s), so only a
//     quotient that is strictly negative gets the sign bit.
// The GPU parity tests sweep every (scale, bf16 value) pair against the CPU oracle.
#pragma once

#include "plq_common.cuh"

namespace plq {
#ifdef __CUDACC__

// two bf16 in one 32-bit word -> float32 (element 0 in the low half)
__device__ __forceinline__ float bf16lo_to_f32(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16hi_to_f32(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// round two float32 to bf16 (nearest even) and return them packed (a in the low half)
__device__ __forceinline__ uint32_t f32x2_to_bf16x2(float a, float b) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(b), "f"(a));
  return d;
}

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// E4M3 code (0..0x7E) -> float32, subnormals included: the code shifted into the float32
// exponent/mantissa position is the value scaled by 2^-120 (a float32 subnormal for codes < 8).
__device__ __forceinline__ float e4m3_code_to_f32(uint32_t c) {
  return __uint_as_float(c << 20) * 1.329227995784916e36f;  // 2^120
}

__device__ __forceinline__ uint32_t f32_to_e4m3_rn_sat(float v) {
  uint16_t d;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(d) : "f"(0.0f), "f"(v));
  return d & 0xFFu;
}

// NVFP4 block scale code from the block's absolute maximum (bf16-valued, >= 0, finite).
__device__ __forceinline__ uint32_t nvfp4_scale_code(float bmax) {
  uint32_t c = f32_to_e4m3_rn_sat(bmax * 0.16666667163372040f);
  const float s = e4m3_code_to_f32(c);
  if (6.0f * s < bmax) c += 1;       // nearest was one step short of the round-up
  c = max(c, 1u);                    // floor 2^-9  (all-zero block -> code 0x01)
  return min(c, 0x7Eu);              // saturate at 448, never the NaN code
}

// Two float32 (bf16-valued) -> two E2M1 codes, the first in bits [0,4); r as in nvfp4_quantize8.
__device__ __forceinline__ uint32_t nvfp4_quantize2(const float2 x, float r) {
  const float2 q = __ffma2_rz(x, make_float2(r, r), make_float2(0.0f, 0.0f));
  uint32_t out;
  asm("{\n\t.reg .b8 b0;\n\tcvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\tmov.b32 %0, {b0, b0, b0, b0};\n\t}"
      : "=r"(out)
      : "f"(q.x), "f"(q.y));
  return out & 0xFFu;
}

// Eight float32 (bf16-valued, four pairs) -> eight E2M1 codes, element 0 in bits [0,4).
__device__ __forceinline__ uint32_t nvfp4_quantize8(const float2* x, float r) {
  float2 q[4];
  const float2 r2 = make_float2(r, r), zero = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int i = 0; i < 4; ++i) q[i] = __ffma2_rz(x[i], r2, zero);
  uint32_t out;
  asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n\t"
      "mov.b32 %0, {b0, b1, b2, b3};\n\t}"
      : "=r"(out)
      : "f"(q[0].x), "f"(q[0].y), "f"(q[1].x), "f"(q[1].y), "f"(q[2].x), "f"(q[2].y), "f"(q[3].x), "f"(q[3].y));
  // No sign fix-up is needed here: the quotient is zero only for x = +-0, and the + 0 of the multiply-add turns a -0
  // product into +0, which is what the reference's sign(x/s) * |q| gives; a negative x that merely rounds to zero
  // keeps its sign.
  return out;
}

// MXFP8 block scale byte (exponent + 127) from the block's absolute maximum (bf16-valued).
__device__ __forceinline__ uint32_t mxfp8_scale_code(float bmax) {
  const uint32_t u = __float_as_uint(bmax);
  const int exp = static_cast<int>(u >> 23);          // biased; sign is 0
  const int man = static_cast<int>((u >> 16) & 0x7F);  // the 7 bf16 mantissa bits
  // max = (1 + man/128) * 2^(exp-127);  448 = 1.75 * 2^8  ->  e = exp-127-8 (+1 if 1+man/128 > 1.75)
  int code = exp - 8 + (man > 96 ? 1 : 0);
  if (exp == 0) code = 1;                              // zero / subnormal max
  return static_cast<uint32_t>(max(code, 1));          // floor 2^-126
}

// Eight float32 (four pairs) -> eight E4M3 bytes (element 0 in the low byte of .x); inv = 2^-e.
// The reference multiplies the rounded magnitude by sign(x / s), so a quotient that is exactly zero must lose
// its sign while a negative one that merely rounds to zero keeps it: fl(x * inv) + (+0) does that (-0 + +0 = +0,
// every other value unchanged); x * inv is exact apart from underflow, where it rounds like the reference's x / s
// (so the product is rounded on its own, not fused with the addition).
__device__ __forceinline__ uint2 mxfp8_quantize8(const float2* x, float inv) {
  uint16_t h[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    // scalar _rn intrinsics: never contracted into one fused multiply-add (which would round the exact tiny
    // product straight to -0 and keep the sign)
    const float q0 = __fadd_rn(__fmul_rn(x[i].x, inv), 0.0f), q1 = __fadd_rn(__fmul_rn(x[i].y, inv), 0.0f);
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(h[i]) : "f"(q1), "f"(q0));
  }
  uint2 out;
  out.x = static_cast<uint32_t>(h[0]) | (static_cast<uint32_t>(h[1]) << 16);
  out.y = static_cast<uint32_t>(h[2]) | (static_cast<uint32_t>(h[3]) << 16);
  return out;
}

// 2^(code-127) as float32 for an E8M0 byte in [1, 254].
__device__ __forceinline__ float e8m0_to_f32(uint32_t code) { return __uint_as_float(code << 23); }

// ---- SiLU ------------------------------------------------------------------------------------
// SiLU(g) = g / (1 + exp(-g)) of a bf16-valued g, to be rounded to bf16 by the caller.  The CPU oracle defines it
// with a float32 exponential written down operation by operation and an IEEE division (silu_mul_bf16 / exp_det); the
// value needed is its rounding to 8 significant bits for one of 65 280 possible inputs, and the hardware's ex2 and
// rcp approximations (a few units in the 24th bit) give the same bf16 for every one of them - two GPU tests compare all
// finite inputs, test_silu_of_every_bf16_value_bit_exact and test_silu_of_the_smallest_values_bit_exact - with 5 instructions per element instead of the definition's ~35 ([32768, 28672] -> packed:
// 2175 -> 890 us = 4.8 TB/s).
// The denominator is scaled by 1/4: up to 2^126 its reciprocal is a normal number, above that exp has overflowed and
// the quotient is zero on either path.
__device__ __forceinline__ float2 silu2(float2 g) {
  const float2 q = make_float2(0.25f, 0.25f);
  const float2 t = __fmul2_rn(g, make_float2(-1.44269502162933349609375f, -1.44269502162933349609375f));
  const float2 d = __ffma2_rn(make_float2(ex2_approx(t.x), ex2_approx(t.y)), q, q);
  return __fmul2_rn(__fmul2_rn(g, q), make_float2(rcp_approx(d.x), rcp_approx(d.y)));
}

#endif  // __CUDACC__
}  // namespace plq
