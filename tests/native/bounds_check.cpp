// Test-only wrapper exposing the host side of amcafe_gb300/csrc/cafe_bounds.h
// beside the double-precision expressions that its functions stand in for. Built
// by tests/test_bounds.py.
#include <stdint.h>

#include "../../amcafe_gb300/csrc/cafe_bounds.h"

extern "C" {
// n slots: offsets c0[3], rotation R[9], direction; bounds and the numerator of
// VoxelsCA.C:409-424.
void bc_glb(long n, double dx, const double *c0, const double *R, const int *dir, float *lo, float *hi, double *g) {
  const double pi4 = 3.14159265358979323846 / 4.0, pi2 = 3.14159265358979323846 / 2.0;
  for (long i = 0; i < n; ++i) {
    const double *c = c0 + 3 * i, *r = R + 9 * i;
    float cf[3], rf[9];
    for (int k = 0; k < 3; ++k) cf[k] = cafe_trunc_f32(c[k]);
    for (int k = 0; k < 9; ++k) rf[k] = cafe_trunc_f32(r[k]);
    cafe_glb_slot(dir[i], cf, (float)dx, rf, lo[i], hi[i]);
    const int d27 = dir[i] < 13 ? dir[i] : dir[i] + 1;
    const double dn[3] = {c[0] + (d27 % 3 - 1) * dx, c[1] + (d27 / 3 % 3 - 1) * dx, c[2] + (d27 / 9 - 1) * dx};
    double th = crm_atan2(fabs(dn[1]), fabs(dn[0]));
    th = th > pi4 ? pi2 - th : th;
    double ph = crm_atan2(crm_pow_half(dn[0] * dn[0] + dn[1] * dn[1]), fabs(dn[2]));
    ph = ph < pi4 ? pi2 - ph : ph;
    double l = 0.0;
    for (int k = 0; k < 3; ++k) l += fabs(r[k] * dn[0] + r[3 + k] * dn[1] + r[6 + k] * dn[2]);
    g[i] = crm_pow_half(crm_cos(th) * crm_sin(ph)) * l;
  }
}
// One row of n cells: the fast class and TempField.C:155-190's. s: cg, sg, hLX0,
// hLX1, lx, ly, lz, dirp, dx, y, z (centres), first x; a1[6]; front.
void bc_class(int n, const double *s, const double *a1, double front, int i0, int *fast, int *exact) {
  float ra1[6];
  for (int k = 0; k < 6; ++k) ra1[k] = (float)(1.0 / a1[k]);
  const double cg = s[0], sg = s[1], h0 = s[2], h1 = s[3], lx = s[4], ly = s[5], lz = s[6], dirp = s[7], dx = s[8], y0 = s[9], zp = s[10];
  const CafeClassStep C = cafe_class_step(ra1, front, dirp, cg, sg, dx, false);
  const CafeClassRow W = cafe_class_row(C, cg, sg, h0, h1, lx, ly, lz, ((double)i0 + .5) * dx - h0, y0 - h1, zp, n);
  for (int x = 0; x < n; ++x) {
    fast[x] = cafe_class_fast(C, W, x);
    const double x0 = ((double)(i0 + x) + .5) * dx;
    const double xp = cg * (x0 - h0) + sg * (y0 - h1) + h0, yp = -sg * (x0 - h0) + cg * (y0 - h1) + h1;
    const double r0 = xp - lx, r1 = yp - ly, r2 = zp - lz;
    bool in;
    if (dirp * r0 > 0) {
      const double q1 = r1 / a1[1], q2 = r2 / a1[2];
      in = (q1 * q1 + q2 * q2 < 1.0) && (fabs(r0) < front);
    } else {
      const double q0 = r0 / a1[3], q1 = r1 / a1[4], q2 = r2 / a1[5];
      in = q0 * q0 + q1 * q1 + q2 * q2 < 1.0;
    }
    exact[x] = zp > lz ? 0 : (in ? 2 : 1);
  }
}
void bc_div(long n, const double *a, const double *v, double *q) {
  for (long i = 0; i < n; ++i) q[i] = cafe_div_by(a[i], v[i], 1.0 / v[i]);
}
// The limit's key, and the keys of the numerators V * lim and V * lim less a
// relative 2^-16.
void bc_limit(long n, const double *lim, double V, int time, unsigned *key, unsigned *at, unsigned *below) {
  for (long i = 0; i < n; ++i) {
    const double d = time ? lim[i] : lim[i] * V, b = d - fabs(d) * 0x1p-16;
    key[i] = cafe_limit_key(lim[i], cafe_f32_down(V), time != 0);
    at[i] = time ? cafe_key32(cafe_f32_bits((float)d), 0x7f800000) : cafe_key32((int)(crm_bits(d) >> 32), 0x7ff00000);
    below[i] = time ? cafe_key32(cafe_f32_bits((float)b), 0x7f800000) : cafe_key32((int)(crm_bits(b) >> 32), 0x7ff00000);
  }
}
}
