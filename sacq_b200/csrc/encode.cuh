// Encoding of quotients to e4m3 or int8, shared by the activation quantizers and the 8-bit weight rows.
#pragma once

#include "common.cuh"

namespace sacq {

// ---- two fp32 operations per instruction (sm_100's f32x2 forms; each half rounds like the scalar operation)
__device__ __forceinline__ uint64_t f32x2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void halves_of(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// A bf16 pair (one 32-bit word) as two fp32 values.
__device__ __forceinline__ float pair_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float pair_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// The divisor of a quantized row: q = encode(z / s) with IEEE division.  A division costs about a dozen
// instructions per element and, with the unpacking around it, bounded every quantizer by instruction issue (17 per
// element).  One s serves a whole row, so its reciprocal is made once, as the sum of two fp32 numbers r + r2, and a
// quotient is fma(z, r, z r2), two elements per instruction.  r is 1/s rounded down, so that r2 is not negative and a
// quotient of zero keeps its sign.  Compared with the division for all 2^23 significands of s and all 128 significands of a
// bf16 dividend: 11 of the 1.07 G quotients differ, by one ulp, none of them next to a value of fewer than 10 significant
// bits, where an encoding changes; for the scales of a quantizer, fp32(bf16 / 448) and fp32(bf16 / 127), none.  (Two residual
// corrections of z RN(1/s), five instructions instead of two and one more for the signs, took the INT8 recipe's expanders
// 1.06 us per 128 x 128 weights.  Locating the quotient between z r(1 - e) and z r(1 + e) and dividing only where the two
// encode differently is not faster: exact ties are common, and every warp met one.)
struct RowDivisor {
  float s, r, r2;
  bool fast;                    // s in 2^-80 .. 2^80: every term that can matter is exact enough; else divide
};
__device__ __forceinline__ RowDivisor row_divisor(float s) {
  RowDivisor d;
  d.s = s;
  d.r = __frcp_rd(s);
  d.r2 = __fdiv_rn(__fmaf_rn(-s, d.r, 1.0f), s);      // the remainder is exact
  d.fast = s > 8.3e-25f && s < 1.2e24f;               // false for inf and NaN
  return d;
}
// z / s of two elements.
__device__ __forceinline__ uint64_t quotient2(uint64_t z, uint64_t r, uint64_t r2) { return fma2(z, r, mul2(z, r2)); }

// Scale of a row from its largest |x|: a NaN maximum fails `> 0` like in the reference's torch.where, so the row
// keeps scale 1 and its NaN elements stay NaN; an infinite maximum gives an infinite scale.  Both divide
// (the elements of the first are not bounded by its scale).
template <bool I8>
__device__ __forceinline__ RowDivisor scale_of(float mx) {
  const bool ordinary = mx > 0.f;
  RowDivisor d = row_divisor(ordinary ? __fdiv_rn(mx, I8 ? 127.0f : kE4M3Max) : 1.0f);
  d.fast = d.fast && ordinary;
  return d;
}

// Two encoded values of one row -> two bytes, by IEEE division.  I8: round-half-to-even to int8 in [-127, 127]
// (quantize_rows(x, 'int8_symmetric'), perrow_a8_candidate_r3.py:17-25); else e4m3.
template <bool I8>
__device__ __forceinline__ uint32_t encode2(float z0, float z1, float s) {
  if constexpr (I8) {
    // round-half-even of the clamped quotient through the add of 1.5 * 2^23 (exact for |q| <= 127):
    // keeps the float -> int conversion off the special-function pipe the division already loads
    const float qa = fminf(fmaxf(__fdiv_rn(z0, s), -127.f), 127.f);
    const float qb = fminf(fmaxf(__fdiv_rn(z1, s), -127.f), 127.f);
    const uint32_t a = (uint32_t)(__float_as_int(__fadd_rn(qa, 12582912.0f)) - 0x4B400000) & 0xffu;
    const uint32_t b = (uint32_t)(__float_as_int(__fadd_rn(qb, 12582912.0f)) - 0x4B400000) & 0xffu;
    return a | (b << 8);
  } else {
    return float2_to_e4m3x2(sat448(__fdiv_rn(z0, s)), sat448(__fdiv_rn(z1, s)));
  }
}

// 2 P bf16 values of one row (P words, P even) -> 2 P bytes.  I8: where d.fast, |z| is at most 127.5 s, so the
// quotient needs no clamp before it is rounded by the add of 1.5 * 2^23.
template <bool I8, int P>
__device__ __forceinline__ void encode_pairs(const uint32_t (&w)[P], const RowDivisor& d, uint32_t (&out)[P / 2]) {
  if (d.fast) {
    const uint64_t r = f32x2(d.r, d.r), r2 = f32x2(d.r2, d.r2), magic = f32x2(12582912.0f, 12582912.0f);
#pragma unroll
    for (int j = 0; j < P / 2; ++j) {
      uint64_t q0 = quotient2(f32x2(pair_lo(w[2 * j]), pair_hi(w[2 * j])), r, r2);
      uint64_t q1 = quotient2(f32x2(pair_lo(w[2 * j + 1]), pair_hi(w[2 * j + 1])), r, r2);
      float a, b, c, e;
      if constexpr (I8) {
        halves_of(add2(q0, magic), a, b);
        halves_of(add2(q1, magic), c, e);
        out[j] = __byte_perm(__byte_perm(__float_as_uint(a), __float_as_uint(b), 0x0040),
                             __byte_perm(__float_as_uint(c), __float_as_uint(e), 0x0040), 0x5410);
      } else {
        halves_of(q0, a, b);
        halves_of(q1, c, e);
        out[j] = float2_to_e4m3x2(a, b) | (float2_to_e4m3x2(c, e) << 16);
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < P / 2; ++j)
      out[j] = encode2<I8>(pair_lo(w[2 * j]), pair_hi(w[2 * j]), d.s) |
               (encode2<I8>(pair_lo(w[2 * j + 1]), pair_hi(w[2 * j + 1]), d.s) << 16);
  }
}

// What the bytes of a recipe's weight row need: the bf16 pair operations (mul, add, min, max round once per half,
// like the fp32 operation followed by a conversion).
struct RowWeights {
  RowDivisor d;
  // |w| is clamped to a bf16 value that encodes to the largest byte, so that a caller's own row scale cannot overflow
  // the quotient.  int8: the largest one below 127.5 times the row scale; it is above 126.5 times it (bf16 values
  // are at most 1/128 apart).  e4m3: about 1,000 times the row scale, which saturates.
  __nv_bfloat162 lim, neg_lim;
};
template <bool I8>
__device__ __forceinline__ RowWeights row_weights(float sw) {
  RowWeights w;
  w.d = row_divisor(sw);
  // a row scale that is not an ordinary number takes the division, which clamps by itself
  const __nv_bfloat16 l = w.d.fast ? __float2bfloat16_rz((I8 ? 127.4999f : 1000.f) * sw) : __ushort_as_bfloat16(0x7f80);
  w.lim = __halves2bfloat162(l, l);
  w.neg_lim = __hneg2(w.lim);
  return w;
}

// 16 weights of one row -> 16 bytes: bf16(bf16(c * s) + shift) divided by the row scale and encoded.  pair: 16
// codebook elements; s2, shift2: the scale and the shift in both halves.  A shift of zero (has_shift false) changes a weight in
// its sign only, where the product is a zero or underflows to one (-0 + 0 = 0).  An int8 has no such sign: one fused instruction.
// e4m3 keeps it, and a fused sum would round a negative product that underflows to -0: two instructions.
template <bool I8>
__device__ __forceinline__ void encode_weights16(const uint32_t (&pair)[8], __nv_bfloat162 s2, __nv_bfloat162 shift2,
                                                 bool has_shift, const RowWeights& r, uint32_t (&out)[4]) {
  uint32_t w[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const __nv_bfloat162 c = *reinterpret_cast<const __nv_bfloat162*>(&pair[j]);
    __nv_bfloat162 v = !I8 || has_shift ? __hadd2_rn(__hmul2_rn(c, s2), shift2) : __hfma2(c, s2, shift2);
    if constexpr (I8) v = __hmin2(__hmax2(v, r.neg_lim), r.lim);
    else v = __hmin2_nan(__hmax2_nan(v, r.neg_lim), r.lim);      // a NaN stays one
    w[j] = *reinterpret_cast<const uint32_t*>(&v);
  }
  encode_pairs<I8, 8>(w, r.d, out);
}

}  // namespace sacq
