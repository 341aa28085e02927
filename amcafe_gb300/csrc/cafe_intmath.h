// exp, division and square root in integer arithmetic, correctly rounded, for
// host and device. This GPU completes one double-precision warp-instruction per
// 64 cycles and sub-partition and an integer one in one or two, so where a kernel
// is bound by FP64 issue these are several times cheaper than the floating-point
// sequences: exp takes no double-precision instruction (crm_exp ~55), a quotient
// none (a division ~12), a square root none (~15).
//
// Every function returns exactly what crm_exp, a / b and sqrt(x) return: the
// quotient and the root are rounded from the exact remainder, exp only when its
// error bound cannot change the rounding; arguments outside the stated ranges,
// and undecided ones, take the floating-point function.
#ifndef CAFE_INTMATH_H
#define CAFE_INTMATH_H

#include <stdint.h>

#include "cafe_crmath.h"

CRM_HD uint64_t crm_mulhi64(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}
#define CRM_MANT_MASK 0xfffffffffffffULL
#define CRM_MANT_ONE 0x10000000000000ULL

// The floating-point functions, out of line.
CRM_COLD double crm_exp_fp(double x) { return crm_exp(x); }
CRM_COLD double crm_div_fp(double a, double b) { return a / b; }
CRM_COLD double crm_sqrt_fp(double x) { return sqrt(x); }

// ------------------------------------------------------------------ exp
// crm_exp(x); the integer path takes x in [-707, -2^-40].
//
// t = |x| log2 e = N + j/128 + v/128 with 64 bits of v, |x| log2 e from the 53-bit
// significand and 95 bits of the constant; exp(x) = 2^-N 2^(-j/128) (1 - p), p = 1 -
// exp(-z), z = v ln 2 / 128 < 2^-7.5, by its series to z^7 with the precision that
// each term needs; the table holds 2^(-j/128) / 2 in 95 bits. Absolute errors of the
// result R / 2 in [1/4, 1/2): t 2^-71 ln 2 / 2, z 2 units and the sum of the series
// 2^-70.2, the product and the table 2^-71: below 2^-69 together; 2^-68 is allowed
// for, which leaves one argument in 2^13 undecided.
CRM_HD double crm_exp_int(double x) {
  const uint64_t b = (uint64_t)crm_bits(x), a = b & (uint64_t)CRM_ABS_MASK;
  const int e = (int)(a >> 52) - 1023;
  if (!(b >> 63) || e < -40 || a > 0x4086180000000000ULL) {  // 707
    if ((b >> 63) && a > 0x4087499999999999ULL && a <= (uint64_t)CRM_BITS_INF) return 0.0;  // below -745.2
    return crm_exp_fp(x);
  }
  const uint64_t m = ((a & CRM_MANT_MASK) | CRM_MANT_ONE) << 11;
  // m log2 e, 128 bits: t 2^(126 - e)
  uint64_t hi = crm_mulhi64(m, CRM_LOG2E_63), lo = m * CRM_LOG2E_63;
  const uint64_t c = (uint64_t)(uint32_t)(m >> 32) * CRM_LOG2E_95;
  lo += c;
  hi += lo < c;
  // (N, j) and 64 bits of v: t 2^71
  const int s = 55 - e;
  uint64_t v;
  if (s < 64) {
    v = (lo >> s) | (hi << (64 - s));
    hi >>= s;
  } else {
    v = hi >> (s - 64);
    hi = 0;
  }
  const int j = (int)hi & 127, N = (int)(hi >> 7);
  // z 2^71, and the series from the inside
  const uint64_t z = crm_mulhi64(v, CRM_LN2_64);
  const uint32_t zh = (uint32_t)(z >> 32);  // z 2^39
  const uint32_t i5 = CRM_R720_40 - (uint32_t)(((uint64_t)zh * CRM_R5040_42) >> 41);
  const uint32_t i4 = CRM_R120_38 - (uint32_t)(((uint64_t)zh * i5) >> 41);
  const uint64_t i3 = 0xaaaaaaaaaaaaaaaULL - (((uint64_t)zh * i4) >> 13);
  const uint64_t i2 = 0x2aaaaaaaaaaaaaaaULL - (crm_mulhi64(z, i3) >> 7);
  const uint64_t i1 = 0x8000000000000000ULL - (crm_mulhi64(z, i2) >> 7);
  const uint64_t sr = ~0ULL - (crm_mulhi64(z, i1) >> 7);
  const uint64_t p = crm_mulhi64(z, sr);  // p 2^71
  const uint64_t th = CRM_TAB(crm_exp2n_tab)[j][0], tl = CRM_TAB(crm_exp2n_tab)[j][1];
  const uint64_t tp = crm_mulhi64(th, p);
  // R/2 in 96 bits
  const uint32_t l0 = (uint32_t)tl, l1 = (uint32_t)(tp & 127u) << 25;
  const uint64_t rh = th - (tp >> 7) - (l0 < l1);
  const uint32_t rl = l0 - l1;
  const uint64_t rem = ((rh & 1023u) << 32) | rl, half = 1ULL << 41, err = 1ULL << 28;
  if ((rh >> 62) != 1u || rem - (half - err) <= 2 * err) return crm_exp_fp(x);
  const uint64_t mant = (rh >> 10) + (rem > half);  // in [2^52, 2^53]
  return crm_from_bits((long long)(((uint64_t)(1021 - N) << 52) + mant));
}

// ------------------------------------------------------------------ division
// The reciprocal of a positive normal divisor b = m 2^(eb - 1075): y = 2^116 / m to
// a few units of its 64 bits, from the single-precision reciprocal by two Newton
// steps. eb < 0: not a positive normal number.
struct crm_recip {
  uint64_t y, m;
  int eb;
};
CRM_HD crm_recip crm_reciprocal(double b) {
  crm_recip R;
  const uint64_t bb = (uint64_t)crm_bits(b);
  const int eb = (int)(bb >> 52);  // (sign included)
  R.eb = eb - 1 < 2046u - 1u && eb > 0 ? eb : -1;
  R.m = (bb & CRM_MANT_MASK) | CRM_MANT_ONE;
  const uint64_t m = R.m << 11;
  const uint32_t mh = (uint32_t)(m >> 32), ml = (uint32_t)m;
  const float f = crm_rcp_f32((float)mh) * 0x1p63f;
  const uint32_t y0 = (uint32_t)(f < 4294967040.0f ? f : 4294967040.0f);  // 2^63 / mh, below 2^32
  // (errors 2^-23, 2^-46, then the units lost below)
  const int64_t d0 = (int64_t)(0x8000000000000000ULL - ((uint64_t)mh * y0 + (((uint64_t)ml * y0) >> 32)));
  const uint64_t y1 = ((uint64_t)y0 << 32) + (uint64_t)(((d0 >> 10) * (int64_t)(uint64_t)y0) >> 21);
  const int64_t d1 = (int64_t)(0x8000000000000000ULL - crm_mulhi64(m, y1));
  const uint64_t y2 = y1 + (uint64_t)(((int64_t)(y1 >> 32) * d1) >> 31);
  R.y = R.m == CRM_MANT_ONE ? ~0ULL : y2;
  return R;
}
// a / (b 2^k), b the number of R.
CRM_HD double crm_quotient(double a, const crm_recip &R, double b, int k) {
  const uint64_t ab = (uint64_t)crm_bits(a), aa = ab & (uint64_t)CRM_ABS_MASK;
  const int ea = (int)(aa >> 52);
  const uint64_t m = (aa & CRM_MANT_MASK) | CRM_MANT_ONE;
  const int lt = m < R.m;
  const int e = ea - R.eb - k + 1023 - lt;
  if (R.eb < 0 || ea == 0 || ea == 2047 || e < 1 || e > 2046) return crm_div_fp(a, b * crm_from_bits((long long)(1023 + k) << 52));
  // q within a few units of 2^-10 of m 2^(52 + lt) / R.m, so that the nearest integer
  // follows from the exact remainder (a tie would need 54 significant bits in m)
  const uint64_t q = crm_mulhi64(m << (10 + lt), R.y) >> 10;
  const int64_t r = (int64_t)((m << (52 + lt)) - q * R.m);
  const uint64_t n = q + (2 * r > (int64_t)R.m);  // in [2^52, 2^53]
  return crm_from_bits((long long)((ab & 0x8000000000000000ULL) | (((uint64_t)(e - 1) << 52) + n)));
}
// a / b.
CRM_HD double crm_div_int(double a, double b) { return crm_quotient(a, crm_reciprocal(b), b, 0); }

// ------------------------------------------------------------------ square root
// Single-precision 1/sqrt(x), a relative 2^-21 at least.
CRM_HD float crm_rsqrt_f32(float x) {
#ifdef __CUDA_ARCH__
  return rsqrtf(x);
#else
  return 1.0f / sqrtf(x);
#endif
}
// sqrt(x): for positive normal x a 53-bit root from the single-precision one by two
// steps with exact remainders (errors 2^-21, 2^-42, then a unit), rounded by the
// last remainder (a root has no ties).
CRM_HD double crm_sqrt_int(double x) {
  const uint64_t b = (uint64_t)crm_bits(x);
  const int eb = (int)(b >> 52);  // (sign included)
  if (eb == 0 || eb >= 2047) return crm_sqrt_fp(x);
  const int odd = (eb & 1) ^ 1;  // exponent eb - 1023 odd
  const uint64_t w = ((b & CRM_MANT_MASK) | CRM_MANT_ONE) << (10 + odd);  // in [1, 4), 2^62
  const uint32_t wh = (uint32_t)(w >> 32);
  const float f = crm_rsqrt_f32((float)wh * 0x1p-30f) * 0x1p31f;
  const uint32_t y = (uint32_t)(f < 2147483520.0f ? f : 2147483520.0f);
  const uint64_t s0 = ((uint64_t)wh * y) >> 32;  // the root, 2^29
  const int64_t e0 = (int64_t)(w - ((s0 * s0) << 4));
  const uint64_t s1 = (s0 << 23) + (uint64_t)(((e0 >> 12) * (int64_t)(uint64_t)y) >> 30);  // 2^52
  const int64_t e1 = (int64_t)((w << 42) - s1 * s1);
  uint64_t q = s1 + (uint64_t)(((e1 >> 32) * (int64_t)(uint64_t)y) >> 52);
  // |q - root| < 2: two steps towards the nearest
  for (int i = 0; i < 2; ++i) {
    const int64_t r = (int64_t)((w << 42) - q * q);
    q += (uint64_t)((r > (int64_t)q) - (r <= -(int64_t)q));
  }
  return crm_from_bits((long long)(((uint64_t)((eb - 1023 - odd) / 2 + 1022) << 52) + q));
}

#endif  // CAFE_INTMATH_H
