// Arithmetic of the Mamba convolution tail (problem 029), shared by the stand-alone kernel and the projection's epilogue.
// The rounding steps are the reference's (kernels/029_mamba_conv1d_with_gating/kernel.cu:211-251): masked input,
// convolution, sigmoid and the product are each rounded to bf16.
#pragma once

#include "ptx_sm100.cuh"

namespace so {

constexpr int kConvTaps = 4;

__device__ __forceinline__ float ex2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float2 bf16x2_to_float2(uint32_t w) {
  return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}
__device__ __forceinline__ uint32_t float2_to_bf16x2(float2 v) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(v.y), "f"(v.x));
  return r;
}
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
// bf16(a * m) for both halves of a packed word; the fp32 product of two bf16 values is exact, so this is the
// single rounding of the eager masked multiply
__device__ __forceinline__ uint32_t mask_mul_bf16x2(uint32_t a, uint32_t m2) { return mul_bf16x2(a, m2); }

// convolution + bias for one position of a channel pair, rounded to bf16 (packed)
__device__ __forceinline__ uint32_t conv_pair(float2 x0, float2 x1, float2 x2, float2 x3, const float2 (&w)[4],
                                              float2 bias) {
  float2 acc = __fmul2_rn(x0, w[0]);
  acc = __ffma2_rn(x1, w[1], acc);
  acc = __ffma2_rn(x2, w[2], acc);
  acc = __ffma2_rn(x3, w[3], acc);
  acc = __fadd2_rn(acc, bias);
  return float2_to_bf16x2(acc);
}

// sigmoid of one value in full relative accuracy at any magnitude: e = 2^(-|x| log2 e) with log2 e split into a
// 16-bit head (its product with an 8-bit bf16 significand is exact in fp32) and a tail applied as a first-order
// factor; 1/(1+e) for x >= 0, e/(1+e) for x < 0.  The magnitude stops at 1024, where e is 0 already: an infinity would
// make the tail's product 0 times infinity.  (A NaN takes some finite sigmoid here and is one again in the product with x.)
__device__ __noinline__ float sigmoid_wide(float x) {
  constexpr float kLog2eHead = 1.44268798828125f;      // 0x3fb8aa00
  constexpr float kLog2eTailLn2 = 4.888495152129525e-06f;  // (log2 e - head) * ln 2
  const float a = fminf(fabsf(x), 1024.f);
  const float e0 = ex2_approx(-a * kLog2eHead);
  const float e = fmaf(e0, -a * kLog2eTailLn2, e0);
  const float r = rcp_approx(1.0f + e);
  return x < 0.f ? e * r : r;
}

// bf16(sigmoid) of the four bf16 values in two packed words (the tail kernel takes a channel pair at two positions, the
// projection's epilogue two channel pairs at one), all four arguments >= -20 and none a NaN, which would reach the other
// three (+infinity does not: its denominator is 1): sigmoid = 1 / (1 + 2^(-x log2 e)) directly; each denominator is below
// 2^30, so the product of the four stays finite and ONE reciprocal of it serves all four (products of the other three
// give each quotient back): 1.25 special-function operations per element instead of 2.
__device__ __forceinline__ void sigmoid_2x2(uint32_t ca, uint32_t cb, uint32_t& sa, uint32_t& sb) {
  constexpr float kNegLog2e = -1.4426950408889634f;
  const float2 scale = make_float2(kNegLog2e, kNegLog2e);
  const float2 ta = __fmul2_rn(bf16x2_to_float2(ca), scale);
  const float2 tb = __fmul2_rn(bf16x2_to_float2(cb), scale);
  const float2 one = make_float2(1.f, 1.f);
  const float2 ya = __fadd2_rn(make_float2(ex2_approx(ta.x), ex2_approx(ta.y)), one);
  const float2 yb = __fadd2_rn(make_float2(ex2_approx(tb.x), ex2_approx(tb.y)), one);
  const float2 pab = __fmul2_rn(ya, yb);        // (ya.x*yb.x, ya.y*yb.y)
  const float inv = rcp_approx(pab.x * pab.y);  // 1 / (all four)
  const float2 rab = make_float2(inv * pab.y, inv * pab.x);  // 1/(ya.x*yb.x), 1/(ya.y*yb.y)
  sa = float2_to_bf16x2(__fmul2_rn(rab, yb));   // 1/ya
  sb = float2_to_bf16x2(__fmul2_rn(rab, ya));   // 1/yb
}
// taps 0..3 of the channels (c, c+1), from conv_weight[c][4] as one 16-byte word
__device__ __forceinline__ void unpack_taps(const uint4& q, float2 (&w)[4]) {
  const float2 wa01 = bf16x2_to_float2(q.x), wa23 = bf16x2_to_float2(q.y);  // channel c, taps 0..3
  const float2 wb01 = bf16x2_to_float2(q.z), wb23 = bf16x2_to_float2(q.w);  // channel c + 1
  w[0] = make_float2(wa01.x, wb01.x);
  w[1] = make_float2(wa01.y, wb01.y);
  w[2] = make_float2(wa23.x, wb23.x);
  w[3] = make_float2(wa23.y, wb23.y);
}
// bf16(conv * sigmoid(conv)) of two packed words
__device__ __forceinline__ void silu_2x2(uint32_t ca, uint32_t cb, bool short_form, uint32_t& ra, uint32_t& rb) {
  uint32_t sa, sb;
  if (short_form) {
    sigmoid_2x2(ca, cb, sa, sb);
  } else {
    const float2 xa = bf16x2_to_float2(ca), xb = bf16x2_to_float2(cb);
    sa = float2_to_bf16x2(make_float2(sigmoid_wide(xa.x), sigmoid_wide(xa.y)));
    sb = float2_to_bf16x2(make_float2(sigmoid_wide(xb.x), sigmoid_wide(xb.y)));
  }
  ra = mul_bf16x2(ca, sa);
  rb = mul_bf16x2(cb, sb);
}
// whether the reference keeps an output under this mask value: at least one half (bf16 bits 0x3f00 .. 0x7f80)
__device__ __forceinline__ bool conv_keeps(uint32_t mask_bits) { return mask_bits - 0x3f00u <= 0x4080u; }

}  // namespace so
