// exp, atan2, cos, sin, division and square root in integer arithmetic, correctly
// rounded, for host and device. This GPU completes one double-precision warp-instruction per
// 64 cycles and sub-partition and an integer one in one or two, so where a kernel
// is bound by FP64 issue these are several times cheaper than the floating-point
// sequences: exp takes no double-precision instruction (crm_exp ~55), a quotient
// none (a division ~12), a square root none (~15).
//
// Every function returns exactly what its floating-point counterpart (crm_exp,
// crm_atan2, crm_cos, crm_sin, a / b, sqrt) returns: the quotient and the root are
// rounded from the exact remainder, the others only when their error bounds cannot
// change the rounding; arguments outside the stated ranges, and undecided ones,
// take the floating-point function.
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
CRM_HD int crm_clz64(uint64_t a) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)a);
#else
  return a ? __builtin_clzll(a) : 64;
#endif
}
// 2^e in single precision, -126 <= e <= 127.
CRM_HD float crm_pow2f(int e) {
#ifdef __CUDA_ARCH__
  return __int_as_float((e + 127) << 23);
#else
  const int b = (e + 127) << 23;
  float f;
  memcpy(&f, &b, sizeof f);
  return f;
#endif
}
#define CRM_BITS_PIO2 0x3ff921fb54442d18LL  // CRM_PIO2_1
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
// 2^127 / m for 2^63 < m < 2^64 to a few of its units, from the single-precision
// reciprocal by two Newton steps (errors 2^-23, 2^-46, then the units lost below).
CRM_HD uint64_t crm_recip64(uint64_t m) {
  const uint32_t mh = (uint32_t)(m >> 32), ml = (uint32_t)m;
  const float f = crm_rcp_f32((float)mh) * 0x1p63f;
  const uint32_t y0 = (uint32_t)(f < 4294967040.0f ? f : 4294967040.0f);  // 2^63 / mh, below 2^32
  const int64_t d0 = (int64_t)(0x8000000000000000ULL - ((uint64_t)mh * y0 + (((uint64_t)ml * y0) >> 32)));
  const uint64_t y1 = ((uint64_t)y0 << 32) + (uint64_t)(((d0 >> 10) * (int64_t)(uint64_t)y0) >> 21);
  const int64_t d1 = (int64_t)(0x8000000000000000ULL - crm_mulhi64(m, y1));
  return y1 + (uint64_t)(((int64_t)(y1 >> 32) * d1) >> 31);
}
// The reciprocal of a positive normal divisor b = m 2^(eb - 1075): y = 2^116 / m.
// eb < 0: not a positive normal number.
struct crm_recip {
  uint64_t y, m;
  int eb;
};
CRM_HD crm_recip crm_reciprocal(double b) {
  crm_recip R;
  const uint64_t bb = (uint64_t)crm_bits(b);
  const int eb = (int)(bb >> 52);  // (sign included)
  R.eb = eb > 0 && eb < 2046 ? eb : -1;  // (room for k = 1)
  R.m = (bb & CRM_MANT_MASK) | CRM_MANT_ONE;
  const uint64_t y = crm_recip64(R.m << 11);
  R.y = R.m == CRM_MANT_ONE ? ~0ULL : y;
  return R;
}
// a / (b 2^k), b the number of R, k 0 or 1.
CRM_HD double crm_quotient(double a, const crm_recip &R, double b, int k) {
  const uint64_t ab = (uint64_t)crm_bits(a), aa = ab & (uint64_t)CRM_ABS_MASK;
  const int ea = (int)(aa >> 52);
  const uint64_t m = (aa & CRM_MANT_MASK) | CRM_MANT_ONE;
  const int lt = m < R.m;
  const int e = ea - R.eb - k + 1023 - lt;
  if (R.eb < 0 || ea == 0 || ea == 2047 || e < 1 || e > 2046) {
    if (R.eb > 0 && aa == 0) return a;
    return crm_div_fp(a, b * crm_from_bits((long long)(1023 + k) << 52));
  }
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
// Single-precision 1/sqrt(x). CUDA states 2 ulp for rsqrtf, a relative 2^-22.
CRM_HD float crm_rsqrt_f32(float x) {
#ifdef __CUDA_ARCH__
  return rsqrtf(x);
#else
  return 1.0f / sqrtf(x);
#endif
}
// The 53-bit root of w 2^42, w in [2^62, 2^64), to nearest (a root has no ties), from
// f, 1/sqrt(w / 2^62) with a relative error d of 2^-21 at most: two steps with exact
// remainders leave 1.5 d^2, then less than two units, and the last remainder decides.
// After the first step the root is off by up to 1.5 2^-42 2^53 = 3072 units and its
// remainder takes 67 bits; that of the root's upper 51 bits takes 63 (and does up to
// d = 2^-20.3).
CRM_HD uint64_t crm_root53(uint64_t w, float f) {
  f *= 0x1p31f;
  const uint32_t y = (uint32_t)(f < 2147483520.0f ? f : 2147483520.0f);
  const uint64_t s0 = ((uint64_t)(uint32_t)(w >> 32) * y) >> 32;  // the root, 2^29
  const int64_t e0 = (int64_t)(w - ((s0 * s0) << 4));
  const uint64_t s1 = (s0 << 21) + (uint64_t)(((e0 >> 12) * (int64_t)(uint64_t)y) >> 32);  // 2^50
  const int64_t e1 = (int64_t)((w << 38) - s1 * s1);
  uint64_t q = (s1 << 2) + (uint64_t)(((e1 >> 30) * (int64_t)(uint64_t)y) >> 50);
  // |q - root| < 2: two steps towards the nearest
  for (int i = 0; i < 2; ++i) {
    const int64_t r = (int64_t)((w << 42) - q * q);
    q += (uint64_t)((r > (int64_t)q) - (r <= -(int64_t)q));
  }
  return q;
}
// sqrt(x), in integers for positive normal x.
CRM_HD double crm_sqrt_int(double x) {
  const uint64_t b = (uint64_t)crm_bits(x);
  const int eb = (int)(b >> 52);  // (sign included)
  if (eb == 0 || eb >= 2047) return crm_sqrt_fp(x);
  const int odd = (eb & 1) ^ 1;  // exponent eb - 1023 odd
  const uint64_t w = ((b & CRM_MANT_MASK) | CRM_MANT_ONE) << (10 + odd);  // in [1, 4), 2^62
  const uint64_t q = crm_root53(w, crm_rsqrt_f32((float)(uint32_t)(w >> 32) * 0x1p-30f));
  return crm_from_bits((long long)(((uint64_t)((eb - 1023 - odd) / 2 + 1022) << 52) + q));
}

// crm_pow_half(x).
CRM_COLD double crm_pow_half_fp(double x) { return crm_pow_half(x); }
CRM_HD double crm_pow_half_int(double x) {
  const uint64_t b = (uint64_t)crm_bits(x);
  return b - CRM_MANT_ONE < 2046ULL << 52 ? crm_sqrt_int(x) : crm_pow_half_fp(x);
}

// ------------------------------------------------------------------ atan2
CRM_COLD double crm_atan2_fp(double y, double x) { return crm_atan2(y, x); }
CRM_COLD double crm_cos_fp(double x) { return crm_cos(x); }
CRM_COLD double crm_sin_fp(double x) { return crm_sin(x); }

// crm_atan2(y, x) for y, x >= 0; the integer path takes ratios down to 2^-37.
//
// With t <= 1 the smaller over the larger and c = k/64 next to it, atan t = atan c +
// atan u, u = (num - c den) / (den + c num): the numerator exactly, the quotient to
// 64 bits (2^-70) and its remainder in single precision (2^-90); the series to u^11
// with 83 bits; the table and pi/2 in 95 bits. The errors add up to less than
// 2^-83 (2^-82 is allowed for). A ratio below 1/128 (k = 0) is scaled by 2^s.
CRM_HD double crm_atan2_int(double y, double x) {
  const uint64_t yb = (uint64_t)crm_bits(y), xb = (uint64_t)crm_bits(x);
  const int swap = yb > xb;
  const uint64_t nb = swap ? xb : yb, db = swap ? yb : xb;
  const int en = (int)(nb >> 52), ed = (int)(db >> 52);
  if (nb == 0 && ed > 0 && ed < 2047) return swap ? CRM_PIO2_1 : 0.0;
  const int dl = ed - en;
  if (en <= 0 || ed >= 2047 || dl > 37) return crm_atan2_fp(y, x);
  const uint64_t mn = (nb & CRM_MANT_MASK) | CRM_MANT_ONE, md = (db & CRM_MANT_MASK) | CRM_MANT_ONE;
  const int s = dl > 7 ? dl - 7 : 0, sl = dl > 7 ? 0 : 7 - dl;
  const float tf = (float)(uint32_t)(mn >> 21) * crm_rcp_f32((float)(uint32_t)(md >> 21));
  const int k = s ? 0 : (int)(tf * crm_pow2f(6 - dl) + 0.5f);
  // u 2^s = 8 X / Y; Y is short of den + c num by lost / 2^dl
  const int64_t X = (int64_t)(mn << sl) - (int64_t)(2 * (uint64_t)k * md);
  const uint64_t ax = (uint64_t)(X < 0 ? -X : X), kn = ((uint64_t)k * mn) << 4;
  const uint64_t Y = (md << 10) + (s ? 0 : kn >> dl);
  const uint32_t lost = s ? 0u : (uint32_t)kn & ((1u << dl) - 1u);
  const int z = (int)(Y >> 63) ^ 1;
  const uint64_t m = Y << z;
  const uint64_t rc = (m << 1) == 0 ? ~0ULL : crm_recip64(m);
  const uint64_t U = crm_mulhi64(ax << 10, rc) << z;  // |u| 2^(70 + s)
  // the quotient's remainder, in units of U
  const uint64_t pl = U * Y;
  const int64_t rh = (int64_t)((ax << 9) - crm_mulhi64(U, Y) - (pl != 0));
  const float rf = (float)rh * 0x1p32f + (float)(uint32_t)((0 - pl) >> 32) -
                   (float)(uint32_t)(U >> 32) * (float)lost * crm_pow2f(-dl);
  const float cf = rf * crm_rcp_f32((float)(uint32_t)(Y >> 32));
  const int64_t c = (int64_t)(int)(cf * 0x1p25f);  // 2^-95
  // u (1 - V), V = w (1/3 - w (1/5 - w (1/7 - w (1/9 - w / 11)))), w = u^2
  const uint64_t W = s < 32 ? crm_mulhi64(U, U) >> (2 * s) : 0;  // w 2^76
  const uint32_t wh = (uint32_t)(W >> 30);                       // w 2^46
  const uint32_t q3 = CRM_R9_32 - (uint32_t)(((uint64_t)wh * CRM_R11_35) >> 49);
  const uint32_t q2 = CRM_R7_34 - (uint32_t)(((uint64_t)wh * q3) >> 44);
  const uint64_t q1 = CRM_R5_64 - (((uint64_t)wh * q2) >> 16);
  const uint64_t q0 = CRM_R3_65 - (crm_mulhi64(W, q1) >> 11);
  const uint64_t P = crm_mulhi64(U, crm_mulhi64(W, q0));  // u V 2^83
  // |atan u| 2^s in 95 fraction bits
  int64_t l = (int64_t)((U & 127) << 25) + c - (int64_t)((P & 0xfffff) << 12);
  uint64_t hi = (U >> 7) - (P >> 20) + (uint64_t)(l >> 32);
  uint32_t lo = (uint32_t)l;
  int ex = s;
  if (s && swap) {
    lo = (lo >> s) | (uint32_t)(hi << (32 - s));
    hi >>= s;
    ex = 0;
  }
  // + atan c, and from pi/2
  if (!s) {
    const uint64_t ah = CRM_TAB(crm_atani_tab)[k][0], al = CRM_TAB(crm_atani_tab)[k][1];
    l = X < 0 ? (int64_t)al - (int64_t)lo : (int64_t)al + (int64_t)lo;
    hi = (X < 0 ? ah - hi : ah + hi) + (uint64_t)(l >> 32);
    lo = (uint32_t)l;
  }
  if (swap) {
    l = (int64_t)CRM_PIO2_95 - (int64_t)lo;
    hi = CRM_PIO2_63 - hi + (uint64_t)(l >> 32);
    lo = (uint32_t)l;
  }
  const int lz = crm_clz64(hi);
  if (lz > 20) return crm_atan2_fp(y, x);
  const uint64_t F = lz ? (hi << lz) | (lo >> (32 - lz)) : hi;
  const uint32_t fl = lo << lz;
  const uint64_t rem = ((F & 2047u) << 32) | fl, half = 1ULL << 42, err = 1ULL << (13 + lz);
  if (rem - (half - err) <= 2 * err) return crm_atan2_fp(y, x);
  const uint64_t mant = (F >> 11) + (rem > half);
  return crm_from_bits((long long)(((uint64_t)(1022 - lz - ex) << 52) + mant));
}

// ------------------------------------------------------------------ cos, sin
// cos(r) for 0 <= r < 101.5/128 given in 95 fraction bits; 0: undecided.
//
// c = j/128 next to r, d = r - c: cos r = cos c - cos c (1 - cos d) - sin c sin d,
// the series to d^6 and d^7, cos c in 95 bits. d and sin d are cut to 71 bits,
// the product to another unit: below 3 2^-71 (2^-69 is allowed for).
CRM_HD int crm_cos_core(uint64_t hi, uint32_t lo, double *out) {
  const int j = (int)((hi + (1ULL << 55)) >> 56);
  const int64_t D = (int64_t)(((hi - ((uint64_t)j << 56)) << 8) | (lo >> 24));  // d 2^71
  uint64_t a = D < 0 ? 0 - (uint64_t)D : (uint64_t)D;
  if (a >> 63) a = ~0ULL >> 1;
  const uint64_t W = crm_mulhi64(a, a);     // d^2 2^78
  const uint32_t wh = (uint32_t)(W >> 30);  // d^2 2^48
  const uint64_t ch = CRM_TAB(crm_cosi_tab)[j][0], cl = CRM_TAB(crm_cosi_tab)[j][1], sn = CRM_TAB(crm_cosi_tab)[j][2];
  // cos c (1 - cos d) 2^77
  const uint64_t t1 = CRM_R24_64 - (((uint64_t)wh * CRM_R720_41) >> 25);
  const uint64_t t0 = 0x8000000000000000ULL - (crm_mulhi64(W, t1) >> 14);
  const uint64_t cq = crm_mulhi64(ch, crm_mulhi64(W, t0));
  // sin c sin |d| 2^71
  const uint32_t b1 = CRM_R120_38 - (uint32_t)(((uint64_t)wh * CRM_R5040_44) >> 54);
  const uint64_t b0 = CRM_R6_64 - (((uint64_t)wh * b1) >> 22);
  const uint64_t sd = crm_mulhi64(sn, a - (crm_mulhi64(a, crm_mulhi64(W, b0)) >> 14));
  const int64_t s0 = (int64_t)((sd & 255) << 24);
  const int64_t l = (int64_t)cl - (int64_t)((cq & 0x3fff) << 18) + (D < 0 ? s0 : -s0);
  const uint64_t rh = ch - (cq >> 14) + (D < 0 ? sd >> 8 : 0 - (sd >> 8)) + (uint64_t)(l >> 32);
  const uint64_t rem = ((rh & 1023u) << 32) | (uint32_t)l, half = 1ULL << 41, err = 1ULL << 26;
  *out = crm_from_bits((long long)((1021ULL << 52) + (rh >> 10) + (rem > half)));
  return (rh >> 62) == 1u && rem - (half - err) > 2 * err;
}
// crm_cos(x); the integer path takes x in [0, pi/4].
CRM_HD double crm_cos_int(double x) {
  const uint64_t b = (uint64_t)crm_bits(x);
  if (b > (uint64_t)CRM_BITS_PIO4) return crm_cos_fp(x);
  const int sh = 1023 - (int)(b >> 52);
  if (sh > 27) return 1.0;  // x^2/2 below a quarter ulp of 1
  const uint64_t m = ((b & CRM_MANT_MASK) | CRM_MANT_ONE) << 11;
  double v;
  if (crm_cos_core(m >> sh, (uint32_t)((m << (64 - sh)) >> 32), &v)) return v;
  return crm_cos_fp(x);
}
// crm_sin(x); the integer path takes x in [pi/4, pi/2], as cos(pi/2 - x).
CRM_HD double crm_sin_int(double x) {
  const uint64_t b = (uint64_t)crm_bits(x);
  if (b < (uint64_t)CRM_BITS_PIO4 || b > (uint64_t)CRM_BITS_PIO2) return crm_sin_fp(x);
  const uint64_t m = ((b & CRM_MANT_MASK) | CRM_MANT_ONE) << 11;
  double v;
  if (crm_cos_core(CRM_PIO2_63 - (m >> (1023 - (int)(b >> 52))), (uint32_t)CRM_PIO2_95, &v)) return v;
  return crm_sin_fp(x);
}

#endif  // CAFE_INTMATH_H
