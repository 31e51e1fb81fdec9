/*
 * FP64 operations formed on the integer pipes: products, quotients, square
 * roots and comparisons whose results are those of the IEEE 754 operations
 * (round to nearest, ties to even), bit for bit.
 *
 * GB300 issues FP64 arithmetic at 1/64 of its FP32 rate: one warp-wide FP64
 * instruction holds the SM's FP64 pipe for 16 to 20 cycles, the issue slots
 * of 64 other instructions.  Measured cycles per warp and SM, 32 warps of
 * independent chains: a product here 19.5 (the native one 20.0, but a product
 * here and a native fused multiply-add in turn 22.7 together: the integer
 * pipes are idle while the FP64 pipe works), a quotient by a fixed divisor
 * 18.1 (a native quotient 143.9), a root 43.2 (a native one 150.2).
 *
 * Methods: significands as 64-bit integers with the leading bit at bit 63.
 *   product   a lower bound of the upper product word, normalised; rounding
 *             is decided unless it lies next to a half-way point, where the
 *             native product runs;
 *   quotient  the divisor's 64-bit reciprocal by Newton's iteration from an
 *             FP32 reciprocal, in fixed point, biased low by a few units, so
 *             that the upper product word is a lower bound of the quotient
 *             within 13 units of 2^-64; a quotient of two 53-bit significands
 *             is never half-way between two others, so rounding is decided
 *             unless the bound lies just below a half-way point, where the
 *             sign of the exact remainder of the half-way point decides;
 *   root      1/sqrt by Newton's iteration from an FP32 one, the root
 *             corrected by its residual, and the same treatment of half-way
 *             points.
 * Zero, subnormal, infinite and NaN operands, and results near the ends of
 * the exponent range, take the native operation.
 */
#ifndef RR_FP64_INT_H
#define RR_FP64_INT_H

#include "rr_math.h"

RRM_FN uint64_t fi_mulhi(uint64_t a, uint64_t b) {
#if defined(__CUDA_ARCH__)
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}
/* approximate FP32 reciprocal and reciprocal root, within 2^-22.9 relative; the
 * host's are moved off the correctly rounded value so that tests exercise the
 * iterations */
RRM_FN float fi_rcp_f32(float x) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return nextafterf(1.0f / x, 0.0f);
#endif
}
RRM_FN float fi_rsqrt_f32(float x) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return nextafterf(1.0f / sqrtf(x), 0.0f);
#endif
}
RRM_FN double fi_native_sqrt(double x) {
#if defined(__CUDA_ARCH__)
  return __dsqrt_rn(x);
#else
  return sqrt(x);
#endif
}

#define FI_SIGN 0x8000000000000000ull
RRM_FN uint32_t fi_hi(uint64_t u) { return (uint32_t)(u >> 32); }
RRM_FN int fi_exp(uint64_t u) { return (int)(fi_hi(u) >> 20) & 0x7ff; }
/* the significand of a normal number, leading bit at bit 63 */
RRM_FN uint64_t fi_sig(uint64_t u) { return (u << 11) | FI_SIGN; }
RRM_FN int fi_normal(int e) { return (uint32_t)(e - 1) < 2046u; }
/* sign, biased exponent e (1 .. 2046) and a 53-bit significand, possibly
 * rounded up to 2^53 (the carry moves into the exponent) */
RRM_FN double fi_pack(uint64_t sign, int e, uint64_t sig53) {
  return rrm_from_bits(sign | (sig53 + ((uint64_t)(uint32_t)(e - 1) << 52)));
}

/* a lower bound of floor(a b / 2^64), at most two below it: the three upper
 * partial products, without the carries of the lower ones */
RRM_FN uint64_t fi_mulhi_low(uint64_t a, uint64_t b) {
  const uint64_t x = (uint64_t)fi_hi(a) * (uint32_t)b, y = (uint64_t)(uint32_t)a * fi_hi(b);
  return (uint64_t)fi_hi(a) * fi_hi(b) + fi_hi(x) + fi_hi(y);
}

/* Operand range of an operation with one fixed operand: its other operand's
 * upper word ha is in range when ha * 2 - lo2 <= span2 (unsigned), i.e. its
 * biased exponent lies in [lo, hi]; never, when lo > hi. */
typedef struct {
  uint32_t lo2, span2;
} fi_range;
RRM_FN fi_range fi_range_of(int lo, int hi) {
  fi_range r;
  lo = lo < 1 ? 1 : lo;
  hi = hi > 2046 ? 2046 : hi;
  r.lo2 = lo > hi ? 1u : (uint32_t)lo << 21; /* ha * 2 is even */
  r.span2 = lo > hi ? 0u : ((uint32_t)(hi - lo + 1) << 21) - 1u;
  return r;
}
RRM_FN int fi_in_range(fi_range r, uint32_t ha) { return ha * 2u - r.lo2 <= r.span2; }
/* the double of a 53-bit significand (possibly 2^53) and the rest of its
 * upper word: sign and biased exponent - 1 */
RRM_FN double fi_join(uint64_t sig, uint32_t add) {
  return rrm_from_bits((uint64_t)(fi_hi(sig) + add) << 32 | (uint32_t)sig);
}

/* native operations out of line: a branch to them stays a branch (inlined, the
 * compiler runs the native product for every operand and selects) */
#if defined(__CUDACC__)
#define FI_SLOW static __host__ __device__ __noinline__
#else
#define FI_SLOW static
#endif
FI_SLOW double fi_slow_mul(double a, double b) { return RRM_MUL(a, b); }

/* ---------------------------------------------------------------- product -- */
RRM_FN double fi_mul(double a, double b) {
  const uint64_t ua = rrm_bits(a), ub = rrm_bits(b);
  const int ea = fi_exp(ua), eb = fi_exp(ub), e = ea + eb - 1023;
  uint64_t q = fi_mulhi_low(fi_sig(ua), fi_sig(ub)); /* in [2^62 - 2, 2^64) */
  const int small = (int64_t)q < 0 ? 0 : 1;
  if (small) q += q;
  /* the product's upper bits lie in [q, q + 6); next to a half-way point, and
   * out of the normal range, the native product (a warp in ten) */
  const uint32_t rest = (uint32_t)q & 0x7ffu;
  if (rest - 0x3fau <= 6u || !fi_normal(ea) || !fi_normal(eb) || (uint32_t)(e - 1) >= 2045u) return fi_slow_mul(a, b);
  return fi_pack((ua ^ ub) & FI_SIGN, e + 1 - small, (q >> 11) + (rest >> 10));
}

/* products by one fixed factor */
typedef struct {
  uint64_t sig;
  double b;
  fi_range range;
  uint32_t add;
} fi_factor;
RRM_FN fi_factor fi_factor_of(double b) {
  fi_factor f;
  const uint64_t ub = rrm_bits(b);
  const int eb = fi_exp(ub);
  f.sig = fi_sig(ub);
  f.b = b;
  f.range = fi_range_of(fi_normal(eb) ? 1024 - eb : 1, fi_normal(eb) ? 3068 - eb : 0);
  f.add = ((uint32_t)(eb - 1023) << 20) + (fi_hi(ub) & 0x80000000u);
  return f;
}
RRM_FN double fi_mul_by(double a, fi_factor f) {
  const uint64_t ua = rrm_bits(a);
  const uint32_t ha = fi_hi(ua);
  uint64_t q = fi_mulhi_low(fi_sig(ua), f.sig);
  uint32_t add = (ha & 0xfff00000u) + f.add;
  if ((int64_t)q >= 0) {
    q += q;
    add -= 0x00100000u;
  }
  if (((uint32_t)q << 21) - (0x3fau << 21) < (7u << 21) || !fi_in_range(f.range, ha)) return fi_slow_mul(a, f.b);
  return fi_join((q >> 11) + (((uint32_t)q >> 10) & 1u), add);
}

/* --------------------------------------------------------------- quotient -- */
/* r with 2^127 / D - 4 < r < 2^127 / D - 1 for D in [2^63, 2^64) */
RRM_FN uint64_t fi_recip64(uint64_t D) {
  /* R0 ~ 2^94 / D within 2^-22, below 2^31 */
  const float f = fi_rcp_f32((float)(uint32_t)(D >> 40)); /* in (2^-24, 2^-23] */
  uint32_t R0 = (uint32_t)(f * 0x1p54f);
  R0 = R0 > 0x7fffffffu ? 0x7fffffffu : R0;
  /* e = (2^94 - D R0) / 2^30, |e| <= 2^42 */
  const uint64_t w0 = (uint64_t)(uint32_t)D * R0;
  const uint64_t w1 = (uint64_t)fi_hi(D) * R0 + (w0 >> 32);
  const int64_t e = -(int64_t)((w1 << 2) | (uint64_t)((uint32_t)w0 >> 30));
  /* R1 ~ 2^127 / D within 2^-43.9 */
  const uint64_t R1 = ((uint64_t)R0 << 33) + (uint64_t)(((int64_t)(int32_t)R0 * (int32_t)(e >> 12)) >> 19);
  /* E = (2^127 - D R1) / 2^32, |E| < 2^52 */
  const uint64_t ph = fi_mulhi(D, R1), pl = D * R1;
  const int64_t E = -(int64_t)((ph << 32) | (pl >> 32));
  return R1 + (uint64_t)((((int64_t)(int32_t)(R1 >> 33) * (int32_t)(E >> 21)) >> 41) - 2);
}

/* quotients by one fixed divisor */
typedef struct {
  uint64_t R;  /* fi_recip64 of its significand */
  double b;
  fi_range range;
  uint32_t add;
} fi_divisor;
RRM_FN fi_divisor fi_divisor_of(double b) {
  fi_divisor d;
  const uint64_t ub = rrm_bits(b);
  const int eb = fi_exp(ub);
  d.R = fi_recip64(fi_sig(ub));
  d.b = b;
  d.range = fi_range_of(fi_normal(eb) ? eb - 1021 : 1, fi_normal(eb) ? eb + 1023 : 0);
  d.add = ((uint32_t)(1022 - eb) << 20) + (fi_hi(ub) & 0x80000000u);
  return d;
}
/* operands out of range: a zero over a normal number is a zero, the others
 * take the native operations (out of line: rare, and long where inlined) */
FI_SLOW double fi_slow_div(double a, double b) {
  const uint64_t ua = rrm_bits(a), ub = rrm_bits(b);
  if ((ua << 1) == 0 && fi_normal(fi_exp(ub))) return rrm_from_bits((ua ^ ub) & FI_SIGN);
  return RRM_DIV(a, b);
}
/* the rounded 53-bit significand of a / b for a in range; *add gets the rest
 * of the upper word */
RRM_FN uint64_t fi_quot(uint64_t ua, const fi_divisor* d, uint32_t* add) {
  /* the quotient lies in [q, q + 13) after the shift */
  uint64_t q = fi_mulhi_low(fi_sig(ua), d->R);
  uint32_t s = (fi_hi(ua) & 0xfff00000u) + d->add;
  const int small = (int64_t)q >= 0;
  if (small) {
    q += q;
    s -= 0x00100000u;
  }
  *add = s;
  const uint64_t sig = q >> 11;
  uint32_t up = ((uint32_t)q >> 10) & 1u;
  if (((uint32_t)q << 21) - (0x3f2u << 21) < (0xeu << 21)) {
    /* just below half-way: up when A 2^(53 + small) > (2 sig + 1) D, on 53-bit
     * significands; the difference is far below 2^63 */
    const uint64_t ma = (ua & 0x000fffffffffffffull) | 0x0010000000000000ull;
    const uint64_t mb = (rrm_bits(d->b) & 0x000fffffffffffffull) | 0x0010000000000000ull;
    up = (int64_t)((ma << (53 + small)) - (2 * sig + 1) * mb) > 0 ? 1u : 0u;
  }
  return sig + up;
}
RRM_FN double fi_div_by(double a, const fi_divisor* d) {
  const uint64_t ua = rrm_bits(a);
  if (!fi_in_range(d->range, fi_hi(ua))) return fi_slow_div(a, d->b);
  uint32_t add;
  const uint64_t sig = fi_quot(ua, d, &add);
  return fi_join(sig, add);
}

RRM_FN double fi_div(double a, double b) {
  const fi_divisor d = fi_divisor_of(b);
  return fi_div_by(a, &d);
}

/* f (a / b), both operations rounded: the quotient's significand goes on
 * without being packed.  range: where both results are normal. */
typedef struct {
  fi_divisor d;
  double f;
  uint64_t sig;
  fi_range range;
  uint32_t add;
} fi_scaled;
RRM_FN fi_scaled fi_scaled_of(double f, double b) {
  fi_scaled s;
  const uint64_t uf = rrm_bits(f), ub = rrm_bits(b);
  const int ef = fi_exp(uf), eb = fi_exp(ub);
  const int ok = fi_normal(ef) && fi_normal(eb);
  s.d = fi_divisor_of(b);
  s.f = f;
  s.sig = fi_sig(uf);
  /* quotient exponent ea - eb + 1023, or one below, in [1, 2046] and in the factor's range */
  const int lo = 1024 - ef > 1 ? 1024 - ef : 1, hi = 3068 - ef < 2046 ? 3068 - ef : 2046;
  s.range = fi_range_of(ok ? eb - 1022 + lo : 1, ok ? eb - 1023 + hi : 0);
  s.add = ((uint32_t)(ef - 1022) << 20) + (fi_hi(uf) & 0x80000000u);
  return s;
}
FI_SLOW double fi_slow_scaled(double f, double a, double b) { return RRM_MUL(f, fi_slow_div(a, b)); }
RRM_FN double fi_scaled_quot(double a, const fi_scaled* s) {
  const uint64_t ua = rrm_bits(a);
  uint32_t add;
  const uint64_t sig = fi_quot(ua, &s->d, &add);
  if (!fi_in_range(s->range, fi_hi(ua)) || (sig >> 53) != 0) return fi_slow_scaled(s->f, a, s->d.b);
  uint64_t q = fi_mulhi_low(sig << 11, s->sig);
  uint32_t add2 = add + s->add;
  if ((int64_t)q >= 0) {
    q += q;
    add2 -= 0x00100000u;
  }
  if (((uint32_t)q << 21) - (0x3fau << 21) < (7u << 21)) return fi_slow_mul(s->f, fi_join(sig, add));
  return fi_join((q >> 11) + (((uint32_t)q >> 10) & 1u), add2);
}

/* ------------------------------------------------------------------- root -- */
RRM_FN double fi_sqrt(double x) {
  const uint64_t u = rrm_bits(x);
  const int ex = fi_exp(u);
  if ((u & FI_SIGN) || !fi_normal(ex)) return fi_native_sqrt(x);
  /* x = m 4^h with m in [1, 4), M = m 2^62; y = 1 / sqrt(m) */
  const int odd = (ex & 1) ^ 1; /* the unbiased exponent's parity */
  const uint64_t M = fi_sig(u) >> (1 - odd);
  /* Y0 ~ y 2^31 within 2^-21.9 */
  uint32_t Y0 = (uint32_t)(fi_rsqrt_f32((float)(uint32_t)(M >> 40)) * 0x1p42f);
  Y0 = Y0 > 0x7fffffffu ? 0x7fffffffu : Y0;
  /* e = (1 - m y^2) 2^60 (up to one unit high, |e| < 2^40); Y ~ y 2^63 within
   * 2^-43, lowered by 16 units so that it stays below */
  const int64_t e = (int64_t)(0x1000000000000000ull - fi_mulhi(M, (uint64_t)Y0 * Y0));
  const uint64_t Y = ((uint64_t)Y0 << 32) + (uint64_t)(((int64_t)(int32_t)Y0 * (int32_t)(e >> 9)) >> 20) - 16;
  /* S ~ sqrt(m) 2^61 from below; its residual m 2^122 - S^2 (below 2^82) from
   * bit 32 on, and the correction residual / (2 S) = K y 2^-30 */
  uint64_t S = fi_mulhi(M, Y);
  const uint64_t sh = fi_mulhi(S, S), sl = S * S, ml = M << 60;
  const uint64_t rh = (M >> 4) - sh - (ml < sl ? 1u : 0u);
  const uint64_t K = (rh << 32) | ((ml - sl) >> 32);
  S += ((uint64_t)(uint32_t)(K >> 18) * fi_hi(Y)) >> 43;
  /* the root lies in [S, S + 2) */
  const uint64_t sig = S >> 9;
  const uint32_t rest = (uint32_t)S & 0x1ffu;
  uint32_t up = rest >> 8;
  if (rest - 0xfeu < 2u) up = (int64_t)((M << 44) - (2 * sig + 1) * (2 * sig + 1)) > 0 ? 1u : 0u;
  return fi_pack(0, (ex - 1023 - odd) / 2 + 1023, sig + up);
}

/* ------------------------------------------------------------ comparisons -- */
RRM_FN int fi_isnan(uint64_t u) { return (u & ~FI_SIGN) > 0x7ff0000000000000ull; }
/* order of non-NaN values as integers (both zeros 0) */
RRM_FN int64_t fi_key(uint64_t u) { return (int64_t)u < 0 ? -(int64_t)(u & ~FI_SIGN) : (int64_t)u; }
RRM_FN int fi_lt(double a, double b) {
  const uint64_t ua = rrm_bits(a), ub = rrm_bits(b);
  return !fi_isnan(ua) && !fi_isnan(ub) && fi_key(ua) < fi_key(ub);
}
RRM_FN int fi_eq(double a, double b) {
  const uint64_t ua = rrm_bits(a), ub = rrm_bits(b);
  return !fi_isnan(ua) && !fi_isnan(ub) && fi_key(ua) == fi_key(ub);
}

#endif
