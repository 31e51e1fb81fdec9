/*
 * rr_sin, rr_cos, rr_log and rr_exp of rr_math.h in forms with fewer FP64
 * instructions: every rounded operation that the result depends on is the
 * same one on the same operands, so the results are the same bits (checked on
 * the host and on the device).  What is not such an operation moves to the
 * integer pipes: range and sign tests, the quadrant, conversions from
 * integers, halving.  In sin and cos the two polynomials share one Horner
 * chain whose coefficients each lane picks by its quadrant (a warp holds both
 * kinds of quadrant, so two branches would both run), and the terms in the
 * reduced tail, which is zero below 2^20, are left out.  FP64-pipe
 * instructions per warp, counted in the source: sin and cos 44 before, 21 now;
 * log 30 before on a warp with negative arguments, 20 now.
 */
#ifndef RR_MATH_SPLIT_H
#define RR_MATH_SPLIT_H

#include "fp64_int.h"

#if defined(__CUDACC__)
#define RRS_SLOW static __host__ __device__ __noinline__
#else
#define RRS_SLOW static
#endif

RRS_SLOW double rrs_sincos_large(double x, int shift) { return shift ? rr_cos(x) : rr_sin(x); }

/* sin(x) (shift 0) or cos(x) (shift 1) */
RRM_FN double rrs_sincos(double x, int shift) {
  const uint64_t u = rrm_bits(x), ua = u & ~FI_SIGN;
  if (fi_hi(ua) >= 0x41300000u) { /* |x| >= 2^20, inf or NaN */
    if (ua > 0x7ff0000000000000ull) return x;
    return ua == 0x7ff0000000000000ull ? rrm_nan() : rrs_sincos_large(x, shift);
  }
  const double ax = rrm_from_bits(ua);
  const double t = RRM_ADD(RRM_MUL(ax, 0x1.45f306dc9c883p-1), 0x1.8p52);
  double kd = RRM_SUB(t, 0x1.8p52);
  int q = (int)(uint32_t)rrm_bits(t);
  if (ua <= 0x3fe921fb54442d18ull) { /* |x| <= pi/4: not reduced */
    kd = 0.0;
    q = 0;
  }
  q += shift;
  double r = RRM_FMA(-kd, 0x1.921fb54400000p+0, ax);
  r = RRM_FMA(-kd, 0x1.0b4611a600000p-34, r);
  r = RRM_FMA(-kd, 0x1.3198a2e037073p-69, r);
  const int c = q & 1; /* a cosine of r */
  const double z = RRM_MUL(r, r);
  double p = c ? 0x1.e542ba4020225p-62 : -0x1.2f49b46814157p-57;
  p = RRM_FMA(p, z, c ? -0x1.6827863b97d97p-53 : 0x1.952c77030ad4ap-49);
  p = RRM_FMA(p, z, c ? 0x1.ae7f3e733b81fp-45 : -0x1.ae7f3e733b81fp-41);
  p = RRM_FMA(p, z, c ? -0x1.93974a8c07c9dp-37 : 0x1.6124613a86d09p-33);
  p = RRM_FMA(p, z, c ? 0x1.1eed8eff8d898p-29 : -0x1.ae64567f544e4p-26);
  p = RRM_FMA(p, z, c ? -0x1.27e4fb7789f5cp-22 : 0x1.71de3a556c734p-19);
  p = RRM_FMA(p, z, c ? 0x1.a01a01a01a01ap-16 : -0x1.a01a01a01a01ap-13);
  p = RRM_FMA(p, z, c ? -0x1.6c16c16c16c17p-10 : 0x1.1111111111111p-7);
  p = RRM_FMA(p, z, c ? 0x1.5555555555555p-5 : -0x1.5555555555555p-3);
  /* sin r = r + (r z) p; cos r = h + ((z z) p + ((1 - h) - w)), w = z/2, h = 1 - w */
  double head = r, tail = 0.0;
  if (c) {
    const uint64_t zb = rrm_bits(z);
    const double w = rrm_from_bits(fi_hi(zb) >= 0x00200000u ? zb - 0x0010000000000000ull : zb); /* tiny: h = 1 either way */
    head = RRM_SUB(1.0, w);
    tail = RRM_SUB(RRM_SUB(1.0, head), w);
  }
  const double v = RRM_ADD(head, RRM_FMA(RRM_MUL(z, c ? z : r), p, tail));
  return rrm_from_bits(rrm_bits(v) ^ ((uint64_t)(uint32_t)(q & 2) << 62) ^ (shift ? 0 : u & FI_SIGN));
}
RRM_FN double rrs_sin(double x) { return rrs_sincos(x, 0); }
RRM_FN double rrs_cos(double x) { return rrs_sincos(x, 1); }

/* (double)e for |e| < 2^24, through the float with the same value */
RRM_FN double rrs_int(int e) {
  const float f = (float)e;
  uint32_t b;
#if defined(__CUDA_ARCH__)
  b = __float_as_uint(f);
#else
  memcpy(&b, &f, sizeof b);
#endif
  const uint32_t hi = (b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u);
  return e == 0 ? 0.0 : rrm_from_bits((uint64_t)hi << 32 | (b << 29));
}

RRM_FN double rrs_log(double x) {
  uint64_t b = rrm_bits(x);
  int e = -1023;
  if (b - 0x0010000000000000ull >= 0x7fe0000000000000ull) { /* not a positive normal number */
    if ((b & ~FI_SIGN) > 0x7ff0000000000000ull) return x;
    if ((b << 1) == 0) return -rrm_inf();
    if (b >> 63) return rrm_nan();
    if (b == 0x7ff0000000000000ull) return x;
    b = rrm_bits(RRM_MUL(x, 0x1p54)); /* subnormal */
    e -= 54;
  }
  /* rrm_log_parts with the grid point c and e formed in integers */
  const uint64_t mant = b & 0x000fffffffffffffull;
  e += (int)(b >> 52);
  int j;
  double m, c;
  if (mant > 0x6a09e667f3bccull) {
    m = rrm_from_bits(mant | 0x3fe0000000000000ull);
    e += 1;
    j = (int)((mant + (1ull << 46)) >> 47);
    c = rrm_from_bits(0x3fe0000000000000ull + ((uint64_t)j << 47));
    j -= 32;
  } else {
    m = rrm_from_bits(mant | 0x3ff0000000000000ull);
    j = (int)((mant + (1ull << 45)) >> 46);
    c = rrm_from_bits(0x3ff0000000000000ull + ((uint64_t)j << 46));
  }
  const double invc = RR_LOG_T(j + 19, 0);
  const double f = RRM_SUB(m, c);
  const double rh = RRM_MUL(f, invc);
  const double rl = RRM_MUL(RRM_FMA(-rh, c, f), invc);
  double q = RRM_FMA(rh, RR_LOG_P9, RR_LOG_P8);
  q = RRM_FMA(q, rh, RR_LOG_P7);
  q = RRM_FMA(q, rh, RR_LOG_P6);
  q = RRM_FMA(q, rh, RR_LOG_P5);
  q = RRM_FMA(q, rh, RR_LOG_P4);
  q = RRM_FMA(q, rh, RR_LOG_P3);
  q = RRM_FMA(q, rh, RR_LOG_P2);
  const double tail = RRM_FMA(RRM_MUL(rh, rh), q, rl);
  const double ed = rrs_int(e);
  const double a = RRM_FMA(ed, RR_LOG_LN2_HI, RR_LOG_T(j + 19, 1));
  const double b0 = RRM_FMA(ed, RR_LOG_LN2_LO, RR_LOG_T(j + 19, 2));
  const double s = RRM_ADD(a, rh);
  const double t = RRM_ADD(RRM_SUB(a, s), rh);
  return RRM_ADD(s, RRM_ADD(RRM_ADD(t, tail), b0));
}

RRM_FN double rrs_exp(double x) {
  const uint64_t u = rrm_bits(x), ua = u & ~FI_SIGN;
  if (fi_hi(ua) >= 0x40862000u) { /* |x| >= 708, inf or NaN */
    if (ua > 0x7ff0000000000000ull) return x;
    if (u == ua && ua > 0x40862e42fefa39efull) return rrm_inf(); /* > log(DBL_MAX) */
    if (u != ua && ua > 0x40874910d52d3052ull) return 0.0; /* < log of the least subnormal / 2 */
  }
  return rrm_exp_core(x, 0.0, 0);
}

#endif
