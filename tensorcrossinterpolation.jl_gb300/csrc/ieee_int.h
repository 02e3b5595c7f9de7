// IEEE double multiplication and division on the integer pipes.
//
// GB300 issues one FP64 warp instruction per 64 cycles per SM quarter (77 with
// all four busy), while its integer pipes take one in one to four: a 104 x 104
// rank-1 update in shared memory with two 256-thread CTAs per SM takes 1.20
// cycles per element and SM with multiply and subtract on the FP64 pipe, 0.68
// with the product below and an FP64 subtraction, 0.41 without the subtraction.
// A warp's FP64 division holds its quarter for 548 cycles; int_div takes 118 as
// a chain.
// The results are the correctly rounded ones (nearest, ties to even), bit for
// bit those of __dmul_rn and __ddiv_rn, so pivots and factors do not change.
//
// Both take operands whose exponent keeps the result clear of the subnormal
// range and of overflow: zero, or 2^-510 <= |v| < 2^512 (int_safe).  Callers
// test that and use the FP64 instructions for anything else (Inf, NaN,
// subnormals, extreme magnitudes).
//
// Method: from the definition.  A 53-bit significand is 32 + 21 bits, so its
// product is four 32 x 32 -> 64-bit multiply-adds whose middle sum cannot
// overflow; the top 64 bits and a sticky bit decide the rounding.  A quotient
// of two 53-bit significands is never half way between two doubles, so its
// first 54 bits round it; they come from a multiplication by the divisor's
// 64-bit reciprocal (Newton steps in fixed point from a single-precision
// reciprocal) and one exact remainder.
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define TCI_II __host__ __device__ __forceinline__
#else
#define TCI_II static inline
#endif

#if defined(__CUDA_ARCH__)
TCI_II uint32_t ii_hi(double v) { return (uint32_t)__double2hiint(v); }
TCI_II uint32_t ii_lo(double v) { return (uint32_t)__double2loint(v); }
TCI_II double ii_make(uint32_t hi, uint32_t lo) { return __hiloint2double((int)hi, (int)lo); }
TCI_II uint32_t ii_funnel_r(uint32_t lo, uint32_t hi, uint32_t s) { return __funnelshift_r(lo, hi, s); }
TCI_II uint64_t ii_mulhi(uint64_t a, uint64_t b) { return __umul64hi(a, b); }
TCI_II float ii_float(uint32_t b) { return __uint_as_float(b); }
TCI_II float ii_rcp(float x) {  // within 2 ulp, which the Newton steps absorb
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
#else
TCI_II uint64_t ii_bits(double v) {
  union { double d; uint64_t u; } c;
  c.d = v;
  return c.u;
}
TCI_II uint32_t ii_hi(double v) { return (uint32_t)(ii_bits(v) >> 32); }
TCI_II uint32_t ii_lo(double v) { return (uint32_t)ii_bits(v); }
TCI_II double ii_make(uint32_t hi, uint32_t lo) {
  union { double d; uint64_t u; } c;
  c.u = ((uint64_t)hi << 32) | lo;
  return c.d;
}
TCI_II uint32_t ii_funnel_r(uint32_t lo, uint32_t hi, uint32_t s) {
  return (uint32_t)((((uint64_t)hi << 32) | lo) >> (s & 31));
}
TCI_II uint64_t ii_mulhi(uint64_t a, uint64_t b) { return (uint64_t)(((unsigned __int128)a * b) >> 64); }
TCI_II float ii_float(uint32_t b) {
  union { uint32_t u; float f; } c;
  c.u = b;
  return c.f;
}
TCI_II float ii_rcp(float x) { return 1.0f / x; }
#endif

// Zero, or an exponent field in [513, 1534].
TCI_II bool int_safe(double v) {
  const uint32_t hi = ii_hi(v);
  return ((hi >> 20) & 0x7ffu) - 513u <= 1021u || ((hi << 1) | ii_lo(v)) == 0u;
}

// A factor taken apart: h the top 32 bits of the significand, l the low 21
// (both 0 for a zero), se sign and exponent field in place.
struct IntFactor {
  uint32_t h, l, se;
};
TCI_II IntFactor int_split(double v) {
  const uint32_t hi = ii_hi(v), lo = ii_lo(v);
  IntFactor f;
  f.se = hi & 0xfff00000u;
  const bool zero = (hi << 1) == 0u;  // int_safe: a zero exponent field is a zero
  f.h = zero ? 0u : (((hi << 11) | (lo >> 21)) | 0x80000000u);
  f.l = lo & 0x1fffffu;
  return f;
}

// x * y, both int_safe.
TCI_II double int_mul(const IntFactor& x, const IntFactor& y) {
  const uint64_t t0 = (uint64_t)x.l * y.l;
  uint64_t t1 = (uint64_t)x.h * y.l + (t0 >> 21);
  t1 = (uint64_t)x.l * y.h + t1;  // below 2^55
  const uint64_t T = (uint64_t)x.h * y.h + (t1 >> 21);  // the product's top 64 bits: [2^62, 2^64), or 0
  const uint32_t sticky = (((uint32_t)t1 | (uint32_t)t0) & 0x1fffffu) ? 1u : 0u;
  const uint32_t Th = (uint32_t)(T >> 32), Tl = (uint32_t)T;
  const uint32_t p = Th >> 31, s = 10u + p;
  const uint32_t rl = ii_funnel_r(Tl, Th, s);
  // rest = the bits below the 53 kept ones from the top, sticky and the kept
  // lowest bit at the bottom: above one half, or a tie with an odd result, rounds up
  const uint32_t rest = ((Tl << (22u - p)) | sticky) + (rl & 1u);
  const uint32_t hi = (Th >> s) + (x.se + y.se + ((p << 20) - 0x40000000u));
  const uint64_t r = (((uint64_t)hi << 32) | rl) + (rest > 0x80000000u ? 1u : 0u);
  const uint32_t rh = Th < 0x40000000u ? ((x.se ^ y.se) & 0x80000000u) : (uint32_t)(r >> 32);
  return ii_make(rh, (uint32_t)r);
}

// A factor with at most 25 trailing zero bits in its significand (int_safe, so
// not zero).  Two of them have a product whose lowest set bit lies below the
// half-way bit: never a tie, so rounding needs no sticky and no lowest bit.
// Values computed in floating point nearly always qualify (a zero, an exact 1
// or a small integer does not); int_mul_dense costs half the ALU instructions
// of int_mul: 13 beside the four multiply-adds.
TCI_II bool int_dense(double v) { return (ii_lo(v) & 0x3ffffffu) != 0u; }
struct DenseFactor {
  uint32_t h, l, se;  // the significand left-aligned in 63 bits: 31 and 32 of them
};
TCI_II DenseFactor dense_split(double v) {
  const uint32_t hi = ii_hi(v), lo = ii_lo(v);
  DenseFactor f;
  f.h = (((hi << 10) | (lo >> 22)) & 0x7fffffffu) | 0x40000000u;
  f.l = lo << 10;
  f.se = hi & 0xfff00000u;
  return f;
}
// x * y, both int_safe and int_dense.
TCI_II double int_mul_dense(const DenseFactor& x, const DenseFactor& y) {
  const uint64_t t0 = (uint64_t)x.l * y.l;
  uint64_t t1 = (uint64_t)x.h * y.l + (t0 >> 32);
  t1 += (uint64_t)x.l * y.h;  // below 2^64: h < 2^31, l <= 2^32 - 2^10
  uint64_t T = (uint64_t)x.h * y.h + (t1 >> 32);  // [2^60, 2^62)
  const uint32_t p = (uint32_t)(T >> 61), s = 8u + p;
  T += 128u << p;  // one half of the kept lowest bit
  const uint32_t Th = (uint32_t)(T >> 32), Tl = (uint32_t)T;
  return ii_make((Th >> s) + x.se + y.se + ((p << 20) - 0x40000000u), ii_funnel_r(Tl, Th, s));
}

// A divisor (int_safe, not zero): its 53-bit significand and sign / exponent,
// and R = 2^116 / mant from below, at most 400 units short.
struct IntDivisor {
  uint64_t mant, R;
  uint32_t se;
};
TCI_II IntDivisor int_divisor(double b) {
  IntDivisor d;
  const uint32_t hi = ii_hi(b), lo = ii_lo(b);
  d.se = hi & 0xfff00000u;
  d.mant = ((uint64_t)((hi & 0xfffffu) | 0x100000u) << 32) | lo;
  // with b in [1, 2): r0 ~ 2^31 / b to 2^-22, r1 ~ 2^62 / b to 2^-43, R ~ 2^64 / b
  const uint64_t bq = d.mant << 11;
  const uint32_t bh = (uint32_t)(bq >> 32);
  const uint32_t r0 = (uint32_t)(ii_rcp(ii_float(0x3f800000u | ((bh >> 8) & 0x7fffffu))) * 2147483648.0f);
  const int64_t e0 = (int64_t)((1ull << 62) - (uint64_t)bh * r0);
  const uint64_t r1 = ((uint64_t)r0 << 31) + (uint64_t)(((int64_t)r0 * (int64_t)(int32_t)(e0 >> 10)) >> 21);
  const int64_t e1 = (int64_t)((1ull << 61) - ii_mulhi(bq, r1));
  const uint64_t r2 = (r1 << 2) + (uint64_t)(((int64_t)(r1 >> 31) * e1) >> 28);
  d.R = (d.mant == 1ull << 52) ? ~0ull : r2 - 100u;
  return d;
}

// a / d, a int_safe.
TCI_II double int_div(double a, const IntDivisor& d) {
  const uint32_t hi = ii_hi(a), lo = ii_lo(a);
  const uint32_t se = hi & 0xfff00000u;
  const uint64_t m = ((uint64_t)((hi & 0xfffffu) | 0x100000u) << 32) | lo;
  const uint32_t lt = m < d.mant ? 1u : 0u;
  uint64_t q = ii_mulhi(m << 11, d.R) >> (10u - lt);       // the quotient's first 54 bits, or one less
  const uint64_t rem = (m << (53u + lt)) - q * d.mant;     // modulo 2^64: below 2 mant
  if (rem >= d.mant) q += 1;
  const uint64_t r = ((q + 1) >> 1) + ((uint64_t)(1022u - lt) << 52) + ((uint64_t)(se & 0x7ff00000u) << 32) -
                     ((uint64_t)(d.se & 0x7ff00000u) << 32);
  const uint32_t sign = (se ^ d.se) & 0x80000000u;
  if ((hi << 1) == 0u) return ii_make(sign, 0u);
  return ii_make((uint32_t)(r >> 32) | sign, (uint32_t)r);
}
