/* Test harness for csrc/common/fp64_int.h and rr_math_split.h on the host: the
 * CPU tests compile it with gcc -ffp-contract=off and call it through ctypes. */
#include "../../rils-rols_gb300/csrc/common/rr_math_split.h"

/* op: 0 product, 1 quotient, 2 root, 3 less than, 4 equal, 5 sin, 6 cos, 7 log, 8 exp, 9 product by a fixed factor,
 * 10 y (x / y) and 11 x (y / x) with both roundings; native: the plain form */
void fi_apply(int op, int native, const double* a, const double* b, int64_t n, double* out) {
  for (int64_t i = 0; i < n; ++i) {
    const double x = a[i], y = b[i];
    switch (op) {
      case 0: out[i] = native ? x * y : fi_mul(x, y); break;
      case 1: out[i] = native ? x / y : fi_div(x, y); break;
      case 2: out[i] = native ? sqrt(x) : fi_sqrt(x); break;
      case 3: out[i] = native ? x < y : fi_lt(x, y); break;
      case 4: out[i] = native ? x == y : fi_eq(x, y); break;
      case 5: out[i] = native ? rr_sin(x) : rrs_sin(x); break;
      case 6: out[i] = native ? rr_cos(x) : rrs_cos(x); break;
      case 7: out[i] = native ? rr_log(x) : rrs_log(x); break;
      case 8: out[i] = native ? rr_exp(x) : rrs_exp(x); break;
      case 9: out[i] = native ? x * y : fi_mul_by(x, fi_factor_of(y)); break;
      default: {
        const double f = op == 10 ? y : x, num = op == 10 ? x : y;
        const fi_scaled s = fi_scaled_of(f, op == 10 ? y : x);
        volatile double q = num / (op == 10 ? y : x);
        out[i] = native ? f * q : fi_scaled_quot(num, &s);
        break;
      }
    }
  }
}
