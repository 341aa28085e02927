// Single-precision bounds and decisions of the step kernels, and the division by
// a reciprocal: plain arithmetic, for host and device. None of them changes a
// result: a bound decides only what the double-precision expression would decide
// the same way, and the quotient is the correctly rounded one. Compiled without
// contraction, like the rest.
#ifndef CAFE_BOUNDS_H
#define CAFE_BOUNDS_H

#include "cafe_crmath.h"

// ------------------------------------------------------------------ bit patterns
CRM_HD float cafe_f32_from_bits(int b) {
#ifdef __CUDA_ARCH__
  return __int_as_float(b);
#else
  float f;
  memcpy(&f, &b, sizeof f);
  return f;
#endif
}
CRM_HD int cafe_f32_bits(float f) {
#ifdef __CUDA_ARCH__
  return __float_as_int(f);
#else
  int b;
  memcpy(&b, &f, sizeof b);
  return b;
#endif
}
// x rounded down to single precision.
CRM_HD float cafe_f32_down(double x) {
#ifdef __CUDA_ARCH__
  return __double2float_rd(x);
#else
  const float f = (float)x;
  return (double)f > x ? nextafterf(f, -INFINITY) : f;
#endif
}
// a * b rounded down.
CRM_HD float cafe_mul_down(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fmul_rd(a, b);
#else
  return cafe_f32_down((double)a * (double)b);
#endif
}
// A double in single precision, truncated (no FP64 instruction); zero below the
// normal range, NaN above 2^127.
CRM_HD float cafe_trunc_f32(double x) {
  const long long b = crm_bits(x);
  const int hi = (int)(b >> 32), e = ((hi >> 20) & 0x7ff) - (1023 - 127);
  if (e <= 0) return 0.f;
  if (e >= 255) return cafe_f32_from_bits(0x7fc00000);
  return cafe_f32_from_bits((hi & (int)0x80000000) | ((e << 23) | ((hi & 0xfffff) << 3) | (int)((unsigned)b >> 29)));
}

// ------------------------------------------------------------------ capture numerators
// Bounds of g of the slot in direction `dir` (0..25) of a cell whose centre lies
// at c0 from its octahedron's, rotation R: g = sqrt(cos th sin ph) |R^T dn|_1
// (VoxelsCA.C:409-424), the folded angles in closed form: cos th = max(|dx|, |dy|)
// /rho and sin ph = max(rho, |dz|)/r, both in [1/sqrt 2, 1]. The offsets are good
// to 3e-7 of |c0| plus the cell size (truncation, one product and sum), e is over
// three times that, and R's truncation adds as little; the quotients take the
// errors of both operands, so that offsets that cancel only loosen the bound. R need
// not be a rotation (the axis of an uploaded orientation may have any length): the
// errors of R^T dn grow with its largest entry, those of a rotation's are below one.
// NaN where an operand is not finite.
// rm: one, or the largest magnitude in R where that is more.
CRM_HD void cafe_glb_slot(int dir, const float *c0, float dx, const float *R, float rm, float &lo, float &hi) {
  const float e = 1e-6f * (fabsf(c0[0]) + fabsf(c0[1]) + fabsf(c0[2]) + 3.f * dx);
  const int d27 = dir < 13 ? dir : dir + 1;
  const float a = c0[0] + (float)(d27 % 3 - 1) * dx, b = c0[1] + (float)(d27 / 3 % 3 - 1) * dx,
              c = c0[2] + (float)(d27 / 9 - 1) * dx;
  const float rho2 = a * a + b * b, r2 = rho2 + c * c, rho = sqrtf(rho2);
  const float ct = fmaxf(0.7071f, (fmaxf(fabsf(a), fabsf(b)) - e) / (rho + 1.5f * e));
  const float sp = fmaxf(0.7071f, (fmaxf(rho, fabsf(c)) - 1.5f * e) / (sqrtf(r2) + 2.f * e));
  const float l0 = R[0] * a + R[3] * b + R[6] * c, l1 = R[1] * a + R[4] * b + R[7] * c,
              l2 = R[2] * a + R[5] * b + R[8] * c;
  const float l = fabsf(l0) + fabsf(l1) + fabsf(l2);
  const float el = 8.f * e * rm;
  lo = sqrtf(ct * sp) * fmaxf(l - el, 0.f) * (1.f - 1e-5f);
  hi = (l + el) * (1.f + 1e-5f);
  if (!(r2 < 1e30f) || !(l < 1e30f) || !(e > 1e-20f)) lo = hi = cafe_f32_from_bits(0x7fc00000);  // (fmaxf drops a NaN operand)
}
CRM_HD void cafe_glb_slot(int dir, const float *c0, float dx, const float *R, float &lo, float &hi) {
  float rm = 1.f;
  for (int k = 0; k < 9; ++k) rm = fmaxf(rm, fabsf(R[k]));
  cafe_glb_slot(dir, c0, dx, R, rm, lo, hi);
}

// ------------------------------------------------------------------ temperature class
// The class of TempField.C:155-190 is a test of two or three quotients against
// one; single precision decides it away from the pool's surface.
struct CafeClassStep {
  float du, dw;    // change of the laser-frame coordinates along x
  float i1, i2, i3, i4, i5, imax, front, side;
  bool ok;
};
struct CafeClassRow {
  float u0, w0, r2, eu, amb;
  bool above, usable;
};
// (the sign of dirp r0 is that of the factors unless the product underflows)
CRM_HD CafeClassStep cafe_class_step(const float *ra1, double bmDX0, double dirp, double cg, double sg, double dx0, bool full) {
  CafeClassStep C;
  C.du = (float)(cg * dx0);
  C.dw = (float)(-sg * dx0);
  C.i1 = ra1[1], C.i2 = ra1[2], C.i3 = ra1[3], C.i4 = ra1[4], C.i5 = ra1[5];
  C.imax = fmaxf(fmaxf(fmaxf(fabsf(C.i1), fabsf(C.i2)), fmaxf(fabsf(C.i3), fabsf(C.i4))), fabsf(C.i5));
  C.front = (float)bmDX0;
  C.ok = C.imax < 1e30f && (dirp == 0.0 || fabs(dirp) > 1e-200) && !full;
  C.side = dirp > 0.0 ? 1.f : (dirp < 0.0 ? -1.f : 0.f);
  return C;
}
// A row of n cells along x whose first has its centre at (X + LX/2, Y + LY/2, zp).
// Coordinates relative to the laser are in error by at most eu (roundings to
// single precision of the row's first and along it), quotients by eq.
CRM_HD CafeClassRow cafe_class_row(const CafeClassStep &C, double cg, double sg, double hLX0, double hLX1, double lx, double ly,
                                   double lz, double X, double Y, double zp, int n) {
  CafeClassRow r;
  r.u0 = (float)(cg * X + sg * Y + hLX0 - lx);
  r.w0 = (float)(-sg * X + cg * Y + hLX1 - ly);
  r.r2 = (float)(zp - lz);
  r.above = zp > lz;
  r.eu = 0x1p-21f * (fabsf(r.u0) + fabsf(r.w0) + fabsf(r.r2) + (fabsf(C.du) + fabsf(C.dw)) * (float)n);
  const float eq = r.eu * C.imax;
  r.amb = 16.f * eq + 1e-5f;
  r.usable = C.ok && eq < 0.01f;
  return r;
}
// Class of the row's cell x: 0 (above the laser plane), 1 (outside the pool), 2
// (inside), -1 (undecided: the double-precision test is needed).
CRM_HD int cafe_class_fast(const CafeClassStep &C, const CafeClassRow &r, int x) {
  if (r.above) return 0;
  if (!r.usable) return -1;
  const float u = r.u0 + C.du * (float)x, w = r.w0 + C.dw * (float)x;
  const float du = C.side * u;
  if (!(fabsf(u) > 2.f * r.eu || C.side == 0.f)) return -1;
  const bool ahead = du > 0.f;
  const float q1 = w * (ahead ? C.i1 : C.i4), q2 = r.r2 * (ahead ? C.i2 : C.i5), q0 = ahead ? 0.f : u * C.i3;
  const float d = q0 * q0 + q1 * q1 + q2 * q2;
  if (d > 1.f + r.amb || (ahead && fabsf(u) > C.front + 2.f * r.eu)) return 1;
  if (d < 1.f - r.amb && (!ahead || fabsf(u) < C.front - 2.f * r.eu)) return 2;
  return -1;
}

// ------------------------------------------------------------------ quotients and keys
// a / v for 0 < v normal, y = 1/v correctly rounded: two corrections of a * y by
// the exact remainder (Markstein, IBM J. Res. Dev. 34(1), 1990: with a correctly
// rounded reciprocal the last one rounds the quotient correctly from a faithful
// one). Operands near the ends of the exponent range take the division.
CRM_HD double cafe_div_by(double a, double v, double y) {
  const int ea = (int)((crm_bits(a) >> 52) & 0x7ff), ev = (int)((crm_bits(v) >> 52) & 0x7ff);
  if (ea < 200 || ea > 1800 || ev < 800 || ev > 1200 || (crm_bits(v) & 0xfffffffffffffLL) == 0xfffffffffffffLL)
    return a / v;
  double q = a * y;
  q = fma(fma(-q, v, a), y, q);
  return fma(fma(-q, v, a), y, q);
}
// Order key of the high word of a double, or of a float (exponent mask xm);
// 0xffffffff for inf and NaN.
CRM_HD unsigned int cafe_key32(int hi, int xm) {
  return (hi & xm) == xm ? 0xffffffffu : (unsigned int)(hi ^ ((hi >> 31) | (int)0x80000000));
}
// A key that bounds from below those of all numerators of times at or above lim
// (|lim| < 1e6) less a relative 2^-18, for the velocity Vf, rounded down: keys of
// the numerators' high words, or (time) of the times in single precision. Every
// event's limit is on its chain, and a double-precision operation costs as much
// as ten others: one conversion, then single precision rounded down.
CRM_HD unsigned int cafe_limit_key(double lim, float Vf, bool time) {
  float f = cafe_f32_down(lim);
  if (!time) f = cafe_mul_down(f, Vf);
#ifdef __CUDA_ARCH__
  f = __fmaf_rd(-fabsf(f), 0x1p-17f, f);
#else
  f = cafe_f32_down((double)f - (double)fabsf(f) * 0x1p-17);
#endif
  const int b = cafe_f32_bits(f), e = b >> 23 & 0xff;
  if (e == 255) return 0u;  // (below the range)
  if (time) return cafe_key32(b, 0x7f800000);
  // as the high word of a double; below single precision's normal range the nearest bound
  if (e == 0) return b < 0 ? cafe_key32((int)0xb8100000, 0x7ff00000) : 0x80000000u;
  return cafe_key32((int)((unsigned)b & 0x80000000u) | (((e + 896) << 20 | (b & 0x7fffff) >> 3) + (b < 0 ? 1 : 0)), 0x7ff00000);
}

#endif  // CAFE_BOUNDS_H
