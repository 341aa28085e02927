// Test-only wrapper exposing the host side of amcafe_gb300/csrc/cafe_intmath.h
// beside the floating-point functions. Built by tests/test_intmath.py.
#include "../../amcafe_gb300/csrc/cafe_intmath.h"

extern "C" void ic_eval(int fn, long n, const double *x, const double *y, double *got, double *want) {
  for (long i = 0; i < n; ++i) {
    switch (fn) {
      case 0:
        got[i] = crm_exp_int(x[i]);
        want[i] = crm_exp(x[i]);
        break;
      case 1:
        got[i] = crm_div_int(x[i], y[i]);
        want[i] = x[i] / y[i];
        break;
      case 2:
        got[i] = crm_quotient(x[i], crm_reciprocal(y[i]), y[i], 1);
        want[i] = x[i] / (2 * y[i]);
        break;
      case 4:
        got[i] = crm_atan2(x[i], y[i]);
        want[i] = crm_atan2_acc(x[i], y[i]);
        break;
      case 5:
        got[i] = crm_sin(x[i]);
        want[i] = crm_sin_acc(x[i]);
        break;
      case 6:
        got[i] = crm_cos(x[i]);
        want[i] = crm_cos_acc(x[i]);
        break;
      case 7:
        got[i] = crm_atan2_int(x[i], y[i]);
        want[i] = crm_atan2(x[i], y[i]);
        break;
      case 8:
        got[i] = crm_cos_int(x[i]);
        want[i] = crm_cos(x[i]);
        break;
      case 9:
        got[i] = crm_sin_int(x[i]);
        want[i] = crm_sin(x[i]);
        break;
      case 10:
        got[i] = crm_pow_half_int(x[i]);
        want[i] = crm_pow_half(x[i]);
        break;
      default:
        got[i] = crm_sqrt_int(x[i]);
        want[i] = sqrt(x[i]);
    }
  }
}

// sqrt(x) from a single-precision 1/sqrt that is off by a relative `off`.
extern "C" void ic_root(long n, double off, const double *x, double *got) {
  for (long i = 0; i < n; ++i) {
    int e;
    const double m = frexp(x[i], &e);  // in [1/2, 1)
    const int odd = e & 1;
    const uint64_t w = (uint64_t)(m * 0x1p53) << (odd ? 10 : 11);
    const double f = 1.0 / sqrt((double)w * 0x1p-62) * (1.0 + off);
    got[i] = ldexp((double)crm_root53(w, (float)f), (odd ? e - 1 : e - 2) / 2 - 52);
  }
}
