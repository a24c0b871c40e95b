// Per-token int4 quantiser arithmetic shared by every kernel that produces activation codes
// (the stand-alone quantisers and the decode kernel that quantises in its own prologue), so that
// all of them emit bit-identical scales and codes.
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

namespace dq {

__device__ __forceinline__ float round_to_bf16(float v) {
  unsigned short bits;
  asm("cvt.rn.bf16.f32 %0, %1;" : "=h"(bits) : "f"(v));
  return __uint_as_float(static_cast<uint32_t>(bits) << 16);
}

// Flag in the scale_fp16 argument of the quantisers: codes are written as E4M3 bytes of the same
// integers (the operand format of the FP8-path prefill GEMM) instead of int8.
constexpr int kCodesE4M3 = 0x100;

// scale_fp16 (low byte): 0 = fp32 scale, 1 = scale rounded to fp16, 2 = "bf16 arithmetic": the quantiser as
// torch evaluates it on a bf16 tensor (every intermediate rounded to bf16), which is what the
// reference's PermLinear does when there is neither an activation scale nor an online Hadamard
// (activations/perm_linear.py:131-133 with formats/rtn_int.py:62-67).
__device__ __forceinline__ float token_scale(float amax, int scale_fp16) {
  scale_fp16 &= 0xFF;
  float s = __fdiv_rn(amax, 7.0f);
  if (scale_fp16 == 2) s = round_to_bf16(s);
  if (amax == 0.f) s = 1.0f;
  if (scale_fp16 == 1) {
    s = __half2float(__float2half_rn(fminf(s, 65504.0f)));
    if (s == 0.f) s = 1.0f;
  }
  return s;
}

// clamp(rint(v / s), -8, 7) with v / s correctly rounded, i.e. bit-identical to the IEEE
// division, at a fraction of its instruction count: t = v * (1/s) is within 2 ulp of the true
// quotient, so rint(t) can only differ from rint(v / s) when t lies within a few ulp of a
// half-integer (|t| <= ~7 here, 4 ulp < 4e-6); only those rare elements take the exact division.
// Rounding and the float -> int step avoid the conversion instructions (quarter-rate pipe; at
// prefill sizes this kernel is bound by instruction issue, not by memory): adding and subtracting
// 1.5 * 2^23 rounds to the nearest integer, ties to even, for |t| < 2^22, and the low byte of the
// bit pattern of (q + 1.5 * 2^23) is q as a two's-complement int8.
constexpr float kRoundMagic = 12582912.0f;
// Eight codes at once.  The fast estimate runs for all of them; only if one of them lies within
// reach of a rounding boundary (or the estimate is not finite) does the thread redo all eight with
// the IEEE division - in a branch of its own, so that the division sequence stays out of the
// common path instead of being predicated into it.
__device__ __forceinline__ void quant_codes8(const float* v, float s, float inv_s, float* q) {
  bool exact = false;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float t = __fmul_rn(v[e], inv_s);
    const float qe = __fsub_rn(__fadd_rn(t, kRoundMagic), kRoundMagic);
    const float dist = fabsf(fabsf(__fsub_rn(t, qe)) - 0.5f);
    // the negated comparison also catches a NaN or infinite estimate (1/s overflowed for a denormal
    // scale): t - qe is then NaN.  A finite estimate of any size rounds correctly above (beyond 2^22
    // it is an integer already) and is clamped below.
    exact |= !(dist >= 1e-5f);
    q[e] = fminf(fmaxf(qe, -8.0f), 7.0f);
  }
  if (exact) {
#pragma unroll
    for (int e = 0; e < 8; ++e) q[e] = fminf(fmaxf(rintf(__fdiv_rn(v[e], s)), -8.0f), 7.0f);
  }
}
// The same in bf16 arithmetic: the quotient is rounded to bf16 before it is rounded to an integer.
__device__ __forceinline__ void quant_codes8_bf16(const float* v, float s, float* q) {
#pragma unroll
  for (int e = 0; e < 8; ++e)
    q[e] = fminf(fmaxf(rintf(round_to_bf16(__fdiv_rn(v[e], s))), -8.0f), 7.0f);
}
// four codes in [-8, 7] (as floats) -> four int8 in one word, first code in the low byte
__device__ __forceinline__ uint32_t pack_codes4(float q0, float q1, float q2, float q3) {
  const uint32_t u0 = __float_as_uint(__fadd_rn(q0, kRoundMagic));
  const uint32_t u1 = __float_as_uint(__fadd_rn(q1, kRoundMagic));
  const uint32_t u2 = __float_as_uint(__fadd_rn(q2, kRoundMagic));
  const uint32_t u3 = __float_as_uint(__fadd_rn(q3, kRoundMagic));
  return __byte_perm(__byte_perm(u0, u1, 0x0040), __byte_perm(u2, u3, 0x0040), 0x5410);
}
// the same four codes as E4M3 bytes (integers up to 8 are exact in E4M3; -0 is stored as +0)
__device__ __forceinline__ uint32_t pack_codes4_e4m3(float q0, float q1, float q2, float q3) {
  unsigned short lo, hi;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(lo) : "f"(__fadd_rn(q1, 0.f)), "f"(__fadd_rn(q0, 0.f)));
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(hi) : "f"(__fadd_rn(q3, 0.f)), "f"(__fadd_rn(q2, 0.f)));
  return static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
}


// |a|, |b| and m: the largest, NaN if one of them is.
__device__ __forceinline__ float max3_abs_nan(float m, float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(m), "f"(fabsf(a)), "f"(fabsf(b)));
  return r;
}

// The scale of a row as the code pass needs it.  in_range: no estimate v * inv_s of the row rounds beyond +-7 (the row's
// absmax is its largest: rounding is monotonic), so that no code has to be clamped.  False for a scale that was rounded
// far from absmax / 7 (fp16 overflow or subnormals) and for an infinite row.
struct TokenQuant {
  float s, inv_s;
  bool in_range;
};
__device__ __forceinline__ TokenQuant token_quant(float amax, float s) {
  const float inv_s = __fdiv_rn(1.0f, s);
  return {s, inv_s, __fmul_rn(amax, inv_s) < 7.4f};
}

// Codes of eight values as bytes (int8 or E4M3), the same as quant_codes8 and the pack functions give.  Two elements to an
// instruction, no clamps, one comparison for all eight: the largest distance |t - rint(t)| says whether one lies within
// 1e-5 of a rounding boundary (or is NaN); then, or out of range, all eight take the IEEE division.  An element costs
// three issue slots instead of ten: 8192 rows of 4096 32.8 -> 30.0 us, 8192 of 8192 68.6 -> 58.5, 16384 rows of 4096 across
// 32 heads 28.4 -> 23.1, 2048 rows of 14336 with the Hadamard 86.4 -> 81.5.
__device__ __forceinline__ uint2 quant_pack8(const float* v, const TokenQuant& tq, bool e4m3) {
  float2 r[4], q[4];
  float far = 0.f;
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const float2 t = __fmul2_rn(make_float2(v[2 * p], v[2 * p + 1]), make_float2(tq.inv_s, tq.inv_s));
    r[p] = __fadd2_rn(t, make_float2(kRoundMagic, kRoundMagic));
    q[p] = __fadd2_rn(r[p], make_float2(-kRoundMagic, -kRoundMagic));  // (zero is +0)
    const float2 d = __ffma2_rn(q[p], make_float2(-1.0f, -1.0f), t);
    far = max3_abs_nan(far, d.x, d.y);
  }
  if (!(tq.in_range && far <= 0.49999f)) {
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      q[p].x = fminf(fmaxf(rintf(__fdiv_rn(v[2 * p], tq.s)), -8.0f), 7.0f);
      q[p].y = fminf(fmaxf(rintf(__fdiv_rn(v[2 * p + 1], tq.s)), -8.0f), 7.0f);
      q[p] = __fadd2_rn(q[p], make_float2(0.f, 0.f));
      r[p] = __fadd2_rn(q[p], make_float2(kRoundMagic, kRoundMagic));
    }
  }
  uint32_t w[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (e4m3) {
      unsigned short lo, hi;
      asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(lo) : "f"(q[2 * h].y), "f"(q[2 * h].x));
      asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(hi) : "f"(q[2 * h + 1].y), "f"(q[2 * h + 1].x));
      w[h] = static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
    } else {
      w[h] = __byte_perm(__byte_perm(__float_as_uint(r[2 * h].x), __float_as_uint(r[2 * h].y), 0x0040),
                         __byte_perm(__float_as_uint(r[2 * h + 1].x), __float_as_uint(r[2 * h + 1].y), 0x0040), 0x5410);
    }
  }
  return make_uint2(w[0], w[1]);
}

}  // namespace dq
