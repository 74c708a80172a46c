// Arithmetic of the per-token (AQ_SCALE_TOKEN) activation quantizer, shared by the quantizer
// kernels (aq_quantize.cu) and the decode kernel that quantizes its own activations
// (aq_direct_decode.cu), so that both produce the same integers and scales by construction.
#pragma once

#include "aq_common.cuh"

namespace aq {

// scale of a row from its absolute maximum, and the reciprocal used for the fast path below
__device__ __forceinline__ float token_scale_of(float row_absmax) {
  return fmaxf(__fdiv_rn(row_absmax, 127.0f), 1.0e-12f);
}

// rint(v / scale) with IEEE division semantics at the cost of a multiply: v * (1/scale)
// differs from the correctly rounded quotient by less than 2^-22 * |quotient| < 4e-5 for
// |quotient| <= 128, so both round to the same integer unless the product lies within 1e-4
// of a rounding boundary; only then is the division evaluated.
__device__ __forceinline__ int quantize_token_value(float v, float scale, float inv_scale) {
  const float t = __fmul_rn(v, inv_scale);
  int r = __float2int_rn(t);
  if (fabsf(t - static_cast<float>(r)) > 0.5f - 1.0e-4f || fabsf(t) > 128.0f) r = __float2int_rn(__fdiv_rn(v, scale));
  return max(-127, min(127, r));
}

__device__ __forceinline__ uint32_t pack4(int a, int b, int c, int d) {
  return (static_cast<uint32_t>(a) & 0xffu) | ((static_cast<uint32_t>(b) & 0xffu) << 8) |
         ((static_cast<uint32_t>(c) & 0xffu) << 16) | ((static_cast<uint32_t>(d) & 0xffu) << 24);
}

// Four values -> four int8 codes.  v * inv is rounded to a whole number by adding 1.5 * 2^23 (one
// fused multiply-add; the code is the low byte of the sum), the distance to it by a second one.  The
// callers' inv is 1 / scale to 2^-24 of it (one rounding) and |v / scale| <= 128, so v * inv is off by 2^-17, the
// distance by 2^-26 more and, where `exact` rounds the quotient to FP32 first, that by 2^-18: below 0.5 - 2^-16 the
// code is that of `exact` and lies in its range.  Otherwise (and for NaN) all four go to `exact`.  Every value
// that goes there counts in a launch of two microseconds (with 1e-4 in place of 2^-16: 32 x 5120 bf16 2.5, now 1.9).
// Full-rate instructions only: conversions of floats to integers run at a fraction of the rate and, with the
// compares, clamps and masks of quantize_token_value, bounded the quantizers (8192 x 8192 bf16: 59 us).
template <typename Exact>
__device__ __forceinline__ uint32_t quantize4(float v0, float v1, float v2, float v3, float inv, Exact exact) {
  constexpr float kMagic = 12582912.0f, kClear = 0.5f - 1.0f / 65536.0f;
  const float m0 = __fmaf_rn(v0, inv, kMagic), m1 = __fmaf_rn(v1, inv, kMagic);
  const float m2 = __fmaf_rn(v2, inv, kMagic), m3 = __fmaf_rn(v3, inv, kMagic);
  const float d0 = __fmaf_rn(v0, inv, __fsub_rn(kMagic, m0)), d1 = __fmaf_rn(v1, inv, __fsub_rn(kMagic, m1));
  const float d2 = __fmaf_rn(v2, inv, __fsub_rn(kMagic, m2)), d3 = __fmaf_rn(v3, inv, __fsub_rn(kMagic, m3));
  if (fabsf(d0) <= kClear && fabsf(d1) <= kClear && fabsf(d2) <= kClear && fabsf(d3) <= kClear) {
    const uint32_t lo = __byte_perm(__float_as_uint(m0), __float_as_uint(m1), 0x0040);
    const uint32_t hi = __byte_perm(__float_as_uint(m2), __float_as_uint(m3), 0x0040);
    return __byte_perm(lo, hi, 0x5410);
  }
  return pack4(exact(v0), exact(v1), exact(v2), exact(v3));
}

// Eight fp16 or bf16 values (one 16-byte vector) as floats.
__device__ __forceinline__ void unpack8(const uint4& raw, bool bf16, float (&v)[8]) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (bf16) {
      v[2 * i] = __uint_as_float(w[i] << 16);
      v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    } else {
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
      v[2 * i] = f.x;
      v[2 * i + 1] = f.y;
    }
  }
}

}  // namespace aq
