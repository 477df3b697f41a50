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
// element).  One s serves a whole row, so its correctly rounded reciprocal r is made once and a quotient takes
// residual corrections instead, two elements per instruction: q0 = RN(z r), then q' = RN(q + RN(z - q s) r)
// (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev.
// 34(1), 1990: with r = RN(1/s) and q within one ulp of z / s the residual is exact and q' is RN(z / s)).  The first
// correction brings q within an ulp, the second makes it exact for any s.  (Locating the quotient between z r(1 - e)
// and z r(1 + e) and dividing only where the two encode differently is not faster: scales are quotients of 8-bit
// significands by 127 and 448, so exact ties are common, and every warp met one.)  Checked against the division over
// the whole domain of the activation quantizers: every finite bf16 maximum, both formats, every bf16 value up to it
// (2.1 G quotients each), no byte differs.
struct RowDivisor {
  float s, r;
  bool fast;                    // s in 2^-80 .. 2^80: every residual that can matter is exact; else divide
};
__device__ __forceinline__ RowDivisor row_divisor(float s) {
  RowDivisor d;
  d.s = s;
  d.r = __frcp_rn(s);
  d.fast = s > 8.3e-25f && s < 1.2e24f;               // false for inf and NaN
  return d;
}
// RN(z / s) of two elements.
__device__ __forceinline__ uint64_t quotient2(uint64_t z, uint64_t ns, uint64_t r) {
  uint64_t q = mul2(z, r);
  q = fma2(fma2(q, ns, z), r, q);
  return fma2(fma2(q, ns, z), r, q);
}

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
    const uint64_t ns = f32x2(-d.s, -d.s), r = f32x2(d.r, d.r), magic = f32x2(12582912.0f, 12582912.0f);
#pragma unroll
    for (int j = 0; j < P / 2; ++j) {
      uint64_t q0 = quotient2(f32x2(pair_lo(w[2 * j]), pair_hi(w[2 * j])), ns, r);
      uint64_t q1 = quotient2(f32x2(pair_lo(w[2 * j + 1]), pair_hi(w[2 * j + 1])), ns, r);
      float a, b, c, e;
      if constexpr (I8) {
        halves_of(add2(q0, magic), a, b);
        halves_of(add2(q1, magic), c, e);
        out[j] = __byte_perm(__byte_perm(__float_as_uint(a), __float_as_uint(b), 0x0040),
                             __byte_perm(__float_as_uint(c), __float_as_uint(e), 0x0040), 0x5410);
      } else {
        halves_of(q0, a, b);
        halves_of(q1, c, e);
        // the corrections turn a negative zero into a positive one: the signs come from the dividends
        out[j] = float2_to_e4m3x2(a, b) | (float2_to_e4m3x2(c, e) << 16) |
                 (__byte_perm(w[2 * j], w[2 * j + 1], 0x7531) & 0x80808080u);
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
// codebook elements; s2, shift2: the scale and the shift in both halves.
template <bool I8>
__device__ __forceinline__ void encode_weights16(const uint32_t (&pair)[8], __nv_bfloat162 s2, __nv_bfloat162 shift2,
                                                 const RowWeights& r, uint32_t (&out)[4]) {
  uint32_t w[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    __nv_bfloat162 v = __hadd2_rn(__hmul2_rn(*reinterpret_cast<const __nv_bfloat162*>(&pair[j]), s2), shift2);
    if constexpr (I8) v = __hmin2(__hmax2(v, r.neg_lim), r.lim);
    else v = __hmin2_nan(__hmax2_nan(v, r.neg_lim), r.lim);      // a NaN stays one
    w[j] = *reinterpret_cast<const uint32_t*>(&v);
  }
  encode_pairs<I8, 8>(w, r.d, out);
}

}  // namespace sacq
