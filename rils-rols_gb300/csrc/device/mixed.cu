// Mixed-precision fitness path: solve, probes and helpers.
//
// Same contract as the plain path (tune_constants + fitness of
// rils_rols_cpp.cpp:445-541 for every candidate of a round), different
// arithmetic.  The round's distinct factor programs are evaluated once in
// double-float arithmetic into a factor table and their Gram sums are formed
// per distinct pair
// (ftable.cu); here:
//   probe         double-float and FP64 interpreters on up to kProbeRows rows
//                 per distinct factor: the error estimate and non-finite
//                 patterns (certification input);
//   solve         one warp per candidate: gathers its Gram entries, runs a
//                 symmetric-pivoted Cholesky in FP64 (pivot = largest
//                 remaining column norm, as in column-pivoted QR) with one
//                 step of iterative refinement, applies the drop / snap rules
//                 of rils_rols_cpp.cpp:488-517 and gets the SSE from the Gram
//                 identity or flags the candidate for the residual pass;
//                 ambiguous or ill-conditioned systems are queued for the
//                 FP64 path.
#include <cfloat>
#include <cstdint>

#include "../common/df32.h"
#include "../common/rr_math_split.h"
#include "common.cuh"
#include "dfeval.cuh"
#include "mixed.cuh"
#include "plain.cuh"
#include "reduce.cuh"

namespace rrd {

// ------------------------------------------------------------- probe ----
constexpr int kProbeThreads = 512;

// Scalar FP64 interpreter with the semantics of the plain path (rr_math
// functions); the double-float one is eval_row_df (dfeval.cuh).
template <int MM>
__device__ bool probe_eval64(const uint32_t* code, int len, const double* K, const DevData& ds, int64_t row,
                             double (&f)[MM]) {
  double st[RRG_MAX_STACK];
  double tos = 0.0;
  int sp = 0;
  for (int pc = 0; pc < len; ++pc) {
    const uint32_t w = code[pc];
    const int op = (int)(w & 0xffu);
    const uint32_t arg = w >> 8;
    switch (op) {
      case RRG_OP_LDV: tos = ds.X64[(int64_t)arg * ds.n_pad + row]; break;
      case RRG_OP_LDC: tos = K[arg]; break;
      case RRG_OP_PSV:
        if (sp >= RRG_MAX_STACK) return false;
        st[sp++] = tos;
        tos = ds.X64[(int64_t)arg * ds.n_pad + row];
        break;
      case RRG_OP_PSC:
        if (sp >= RRG_MAX_STACK) return false;
        st[sp++] = tos;
        tos = K[arg];
        break;
      case RRG_OP_SIN:
      case RRG_OP_COS: tos = rrs_sincos(tos, op - RRG_OP_SIN); break;
      case RRG_OP_LN: tos = rrs_log(tos); break;
      case RRG_OP_EXP: tos = rrs_exp(tos); break;
      case RRG_OP_SQRT: tos = fi_sqrt(tos); break;
      case RRG_OP_SQR: tos = fi_mul(tos, tos); break;
      case RRG_OP_EMIT:
#pragma unroll
        for (int s = 0; s < MM; ++s)
          if ((int)arg == s) f[s] = tos;
        sp = 0;
        break;
      default: {
        const int kk = op - RRG_OP_BIN;
        const int base = kk >> 3, src = (kk & 7) >> 1, dir = kk & 1;
        double o;
        if (src == RRG_SRC_S) {
          if (sp <= 0) return false;
          o = st[--sp];
        } else if (src == RRG_SRC_V) {
          o = ds.X64[(int64_t)arg * ds.n_pad + row];
        } else {
          o = K[arg];
        }
        const double a = dir == RRG_DIR_N ? o : tos, b = dir == RRG_DIR_N ? tos : o;
        switch (base) {
          case RRG_ADD: tos = __dadd_rn(a, b); break;
          case RRG_SUB: tos = __dsub_rn(a, b); break;
          case RRG_MUL: tos = fi_mul(a, b); break;
          case RRG_DIV: tos = fi_div(a, b); break;
          case RRG_POW: tos = rr_pow(a, b); break;
          case RRG_LT: tos = fi_lt(a, b) ? 1.0 : 0.0; break;
          case RRG_EQ: tos = fi_eq(a, b) ? 1.0 : 0.0; break;
          case RRG_NE: tos = fi_eq(a, b) ? 0.0 : 1.0; break;
          case RRG_MIN: tos = fi_lt(a, b) ? a : b; break;
          default: tos = fi_lt(b, a) ? a : b; break;
        }
      }
    }
  }
  return true;
}

// Certification: bound on the relative error of the penalised fitness
// (1 + loss)(1 + rmse)(1 + size * cp) caused by the table's evaluation, from
// the per-row bound E on the error of the rebuilt sum (independent of cp).
__device__ double cert_fitness_bound(double sse, double E, double n_d, double sst) {
  if (!(sse >= 0.0) || !(E >= 0.0)) return 1e300;
  const double dsse = 2.0 * sqrt(sse * n_d) * E + n_d * E * E;
  const double loss = sse / sst, rmse = sqrt(sse / n_d);
  const double rl = (dsse / sst) / (1.0 + loss);
  const double rr = (sqrt((sse + dsse) / n_d) - rmse) / (1.0 + rmse);
  return rl + rr;
}

constexpr int kSolveK = kMixedMaxM + 1;
// shared memory of one warp's solve
struct SolveSmem {
  double ent[GramSize<kMixedMaxM>::E];
  double G[kSolveK][kSolveK], L[kSolveK][kSolveK];
  double b[kSolveK], d0[kSolveK], z[kSolveK], coef[kSolveK], root[kSolveK], t[2][kSolveK * kSolveK];
  int32_t piv[kSolveK];
};
// One copy each of a quotient and a root: a lone candidate's solve is bound by
// fetching its instructions.
static __device__ __noinline__ double one_div(double a, double b) { return fi_div(a, b); }
static __device__ __noinline__ double one_sqrt(double a) { return fi_sqrt(a); }
// squared-norm ratio to the largest column below which the reference's
// rank cut (eps^2 ~ 5e-32) cannot be ruled out
constexpr double kCutAbs = 1e-24;

// Symmetric pivoted Cholesky of the leading k x k of S.L, by one warp (pivot =
// largest remaining diagonal, i.e. the largest remaining column norm of the
// design, as column-pivoted QR picks).  A pivot is cut when it is small against
// its own column's norm (the Gram sums cannot resolve it) or so small against
// the largest column that the reference's QR, whose cut is at eps^2 of the
// largest squared norm, may cut it; a badly scaled but independent column is
// kept.  Returns the rank, and the smallest pivot against its column's norm.
__device__ int warp_cholesky(SolveSmem& S, int k, double tol, double maxd, double& min_ratio) {
  const int lane = threadIdx.x & 31;
  if (lane < k) {
    S.d0[lane] = S.L[lane][lane];
    S.piv[lane] = lane;
  }
  __syncwarp();
  min_ratio = 1.0;
#pragma unroll 1
  for (int s = 0; s < k; ++s) {
    int p = s;
#pragma unroll 1
    for (int j = s + 1; j < k; ++j)
      if (fi_lt(S.L[p][p], S.L[j][j])) p = j;
    const double dp = S.L[p][p], dq = S.d0[S.piv[p]];
    if (!(dp > tol * dq) || !(dp > kCutAbs * maxd)) return s;
    __syncwarp();
    if (p != s) {
      if (lane < k) {
        const double v = S.L[s][lane];
        S.L[s][lane] = S.L[p][lane];
        S.L[p][lane] = v;
      }
      __syncwarp();
      if (lane < k) {
        const double v = S.L[lane][s];
        S.L[lane][s] = S.L[lane][p];
        S.L[lane][p] = v;
      }
      if (lane == 0) {
        const int32_t v = S.piv[s];
        S.piv[s] = S.piv[p];
        S.piv[p] = v;
      }
      __syncwarp();
    }
    min_ratio = fmin(min_ratio, one_div(dp, dq));
    const double lss = one_sqrt(dp);
    if (lane >= s && lane < k) S.L[lane][s] = lane == s ? lss : one_div(S.L[lane][s], lss);
    __syncwarp();
    const int r = k - s - 1;
    for (int e = lane; e < r * r; e += 32) {
      const int i = s + 1 + e / r, j = s + 1 + e % r;
      if (j <= i) S.L[i][j] = S.L[j][i] = __fma_rn(-S.L[i][s], S.L[j][s], S.L[i][j]);
    }
    __syncwarp();
  }
  return k;
}

// One warp per candidate: its Gram entries are gathered from the round's
// pair sums (FP64 totals of the double-float partials of the factor table);
// tuned candidates get a symmetric-pivoted Cholesky solve with one
// refinement step.  Every candidate then gets its SSE from the Gram identity
//     SSE = y'y - 2 c'b + c'Gc      (c: coefficients after the drop / snap rules)
// when its bound  u * (y'y + 2|c|'|b| + |c|'|G||c|)  is below pass2_tol * SSE;
// otherwise it is flagged for the residual pass.
// The lanes share the work: entries, rows and bounds one or a few to a lane,
// chains only where the order of a sum asks for one, quotients and roots on the
// integer pipes (fp64_int.h).  One candidate of three factors: 62 us with one
// lane doing all of it, 49 so, 30 with one copy each of quotient and root; eight
// rounds at 1M rows, with the probe: 2.39 -> 2.01 ms.
// Entry layout per candidate (mmax = kMixedMaxM): G_ij for i <= j < mmax,
// then sum f_i, then sum f_i * y; pair index -1 reads 0.
__global__ void __launch_bounds__(128) mixed_solve_kernel(SolveArgs a) {
  __shared__ SolveSmem smem[4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int li = blockIdx.x * 4 + warp;
  if (li >= a.n_list) return;
  SolveSmem& S = smem[warp];
  const int mmax = kMixedMaxM;
  const int Gn = mmax * (mmax + 1) / 2, E = Gn + 2 * mmax;
  const int32_t* po = a.pair_of + (size_t)li * E;
  for (int e = lane; e < E; e += 32) {
    const int32_t p = po[e];
    S.ent[e] = p >= 0 ? a.psum[p] : (p <= -2 ? a.pself[-2 - (int64_t)p] : 0.0);
  }
  __syncwarp();
  const int c = a.list[li];
  const rrg_cand cd = a.b.cands[c];
  const double* ent = S.ent;
  const double yy = a.ds.yy;
  // Relative accuracy of the double-float Gram sums with respect to the sums
  // of the absolute values of their terms: about 5u^2 per product and 3u^2
  // per double-float addition (u = 2^-24) over at most ~90 sequential
  // additions per sum, plus the FP64 sum of the chunk partials: about 4e-13.
  const double kU = 1e-12;
  auto queue_fallback = [&](int why) {  // lane 0
    const int slot = atomicAdd(a.fallback, 1);
    if (slot < a.fallback_cap) a.fallback[1 + slot] = c;
    if (a.reasons) atomicAdd(a.reasons + why, 1u);
  };
  const ProbeOut pr = a.probe[c];
  const double n_d = (double)a.ds.n;
  auto cert_bound = [&](double sse, double E) { return cert_fitness_bound(sse, E, n_d, a.ds.sst); };
  // per-row error bound of factor i: the largest probed deviation with a
  // safety factor (exact maximum when every row was probed)
  const double safety = pr.all_rows ? 1.5 : 8.0;
  auto ferr = [&](int i) { return safety * (double)pr.dev[i] + 1e-12 * (double)pr.rms[i]; };
  if (cd.mode != RRG_TUNED) {
    if (lane != 0) return;
    // yp = f: SSE = y'y - 2 f'y + f'f
    const double ff = ent[0], fs = ent[Gn], fy = ent[Gn + mmax];
    const bool nan = ff != ff || fs != fs || fy != fy;
    const bool inf = !nan && (fabs(ff) > DBL_MAX || fabs(fs) > DBL_MAX || fabs(fy) > DBL_MAX);
    uint32_t confirmed = pr.nan64;
    if (nan && !(confirmed & 1u) && a.nanrow && a.nanrow[c] >= 0 && a.nanrow[c] < a.ds.n) {
      double f64[kMixedMaxM];
#pragma unroll 1
      for (int i = 0; i < kMixedMaxM; ++i) f64[i] = 0.0;
      if (probe_eval64<kMixedMaxM>(a.b.code + cd.code_offset, cd.code_len, a.b.consts, a.ds, a.nanrow[c], f64) &&
          f64[0] != f64[0])
        confirmed |= 1u;
    }
    uint8_t p2 = 0;
    double sse;
    if (pr.bad32 || pr.inf64 || inf || (nan && !(confirmed & 1u))) {
      // the table broke down, FP64 overflows, or a table NaN that the FP64 probe
      // does not confirm: the FP64 path scores it
      queue_fallback(pr.bad32 ? FB_PROBE_NONFINITE
                              : (pr.inf64 ? FB_FP64_INF : (inf ? FB_FP32_OVERFLOW : FB_OTHER_NAN)));
      sse = -1.0;
    } else if (nan || (pr.nan64 & 1u)) {
      sse = __longlong_as_double(0x7ff8000000000000ll);
    } else {
      sse = __dadd_rn(__dsub_rn(yy, __dmul_rn(2.0, fy)), ff);
      const double bound = kU * (yy + 2.0 * sqrt(fabs(ff) * yy) + ff);
      if (!(sse > 0.0 && bound <= a.pass2_tol * sse)) {
        // the residual pass gives the SSE; certified rounds check it after
        p2 = 1;
        if (a.certify) a.cert_e[c] = ferr(0);
        sse = -1.0;
      } else if (a.certify && cert_bound(sse, ferr(0)) > a.cert_tol) {
        queue_fallback(FB_CERT);
        sse = -1.0;
      }
    }
    a.sse1[c] = sse;
    a.pass2[c] = p2;
    a.res[c].rank = 0;
    return;
  }
  const int m = cd.n_factors, k = m + 1;
  for (int e = lane; e < k * k; e += 32) {
    const int i = e / k, j = e % k, lo = i < j ? i : j, hi = i < j ? j : i;
    S.G[i][j] = lo == m ? (double)a.ds.n
                        : hi == m ? ent[Gn + lo] : ent[lo * mmax - lo * (lo - 1) / 2 + hi - lo];
  }
  if (lane < k) S.b[lane] = lane < m ? ent[Gn + mmax + lane] : a.ds.ysum;
  __syncwarp();
  // Non-finite sums: NaN (a domain error in some factor) gives NaN
  // coefficients and so the fitness sentinel, as the reference's QR does;
  // +-inf without NaN (FP32 exponent overflow) is re-solved by the FP64 path.
  bool nan_l = false, inf_l = false;
  for (int e = lane; e < k * k + k; e += 32) {
    const double v = e < k * k ? S.G[e / k][e % k] : S.b[e - k * k];
    nan_l |= v != v;
    inf_l |= fabs(v) > DBL_MAX;
  }
  const bool has_nan = __any_sync(0xffffffffu, nan_l), has_inf = __any_sync(0xffffffffu, inf_l);
  // factors whose own sums are NaN (a domain error on some row); the cross
  // sums of a NaN factor are NaN for every partner, so only the diagonal,
  // the factor sum and the factor-y sum identify it
  bool fnan_l = false, finf_l = false;
  if (lane < m) {
    const double d = S.G[lane][lane], sf = S.G[lane][m], sy = S.b[lane];
    fnan_l = d != d || sf != sf || sy != sy;
    finf_l = !fnan_l && (fabs(d) > DBL_MAX || fabs(sf) > DBL_MAX || fabs(sy) > DBL_MAX);
  }
  uint32_t nanmask = __ballot_sync(0xffffffffu, fnan_l);
  const uint32_t infmask = __ballot_sync(0xffffffffu, finf_l);
  const uint32_t fullmask = (1u << m) - 1u;  // m <= kMixedMaxM
  uint32_t confirmed = pr.nan64;
  if ((nanmask & ~confirmed) && a.nanrow && a.nanrow[c] >= 0 && a.nanrow[c] < a.ds.n) {
    // table NaN outside the probe rows: evaluate the first such row in FP64
    if (lane == 0) {
      double f64[kMixedMaxM];
#pragma unroll 1
      for (int i = 0; i < kMixedMaxM; ++i) f64[i] = 0.0;
      if (probe_eval64<kMixedMaxM>(a.b.code + cd.code_offset, cd.code_len, a.b.consts, a.ds, a.nanrow[c], f64))
#pragma unroll 1
        for (int i = 0; i < m; ++i)
          if (f64[i] != f64[i]) confirmed |= 1u << i;
    }
    confirmed = __shfl_sync(0xffffffffu, confirmed, 0);
  }
  nanmask |= pr.nan64 & fullmask;
  if (pr.bad32 || pr.inf64 || infmask || (nanmask & ~confirmed) ||
      (!nanmask && (has_nan || has_inf))) {
    // the table broke down where FP64 did not, FP64 overflow, FP32 exponent
    // overflow, a table NaN the FP64 probe does not confirm, or a non-finite sum outside
    // the factor columns: the FP64 path scores it
    if (lane == 0) {
      queue_fallback(pr.bad32 ? FB_PROBE_NONFINITE
                              : (pr.inf64 ? FB_FP64_INF : (infmask ? FB_FP32_OVERFLOW : FB_OTHER_NAN)));
      a.sse1[c] = -1.0;
      a.pass2[c] = 0;
      a.res[c].rank = 0;
    }
    return;
  }
  double* out = a.coefs + cd.coef_offset;
  if (nanmask) {
    // A NaN factor column makes the reference's QR return NaN coefficients
    // (the sentinel) unless a rank cut among the other columns happens before
    // the QR reaches it.  Full, well-conditioned rank of the other columns
    // rules that out (well away from a cut: 1e-6 of the column's own norm);
    // otherwise the FP64 path decides.
    const uint32_t use = (fullmask & ~nanmask) | (1u << m);
    const int kk = __popc(use);
    if (lane < kk) S.piv[lane] = __fns(use, 0, lane + 1);
    __syncwarp();
    for (int e = lane; e < kk * kk; e += 32) S.L[e / kk][e % kk] = S.G[S.piv[e / kk]][S.piv[e % kk]];
    __syncwarp();
    double hmax = 0.0, mr;
#pragma unroll 1
    for (int i = 0; i < kk; ++i) hmax = fmax(hmax, S.L[i][i]);
    const bool full = warp_cholesky(S, kk, 1e-6, hmax, mr) == kk;
    if (lane < k) out[lane] = __longlong_as_double(0x7ff8000000000000ll);
    if (lane == 0) {
      if (!full) queue_fallback(FB_NAN_RANK);
      a.sse1[c] = full ? __longlong_as_double(0x7ff8000000000000ll) : -1.0;
      a.pass2[c] = 0;
      a.res[c].rank = 0;
    }
    return;
  }
  // (every sum is finite from here on)
  for (int e = lane; e < k * k; e += 32) S.L[e / k][e % k] = S.G[e / k][e % k];
  if (lane < k) {
    S.root[lane] = one_sqrt(fabs(S.G[lane][lane]));
    S.coef[lane] = 0.0;
  }
  __syncwarp();
  double maxd = 0.0, min_ratio;
#pragma unroll 1
  for (int i = 0; i < k; ++i) maxd = fmax(maxd, S.G[i][i]);
  const int rank = warp_cholesky(S, k, a.rank_tol, maxd, min_ratio);
  // solve L L^T z = P b on the leading `rank` block, then one refinement step
  const int pl = lane < rank ? S.piv[lane] : 0;
  double rhs = lane < rank ? S.b[pl] : 0.0;
#pragma unroll 1
  for (int pass = 0; pass < 2 && rank > 0; ++pass) {
    double v = rhs;  // forward: lane i's row, its terms in the order of the columns
#pragma unroll 1
    for (int j = 0; j < rank; ++j) {
      if (lane == j) v = one_div(v, S.L[j][j]);
      const double zj = __shfl_sync(0xffffffffu, v, j);
      if (lane > j && lane < rank) v = __fma_rn(-S.L[lane][j], zj, v);
    }
    if (lane < rank) S.z[lane] = v;
    __syncwarp();
#pragma unroll 1
    for (int i = rank - 1; i >= 0; --i) {
      double w = S.z[i];
#pragma unroll 1
      for (int j = i + 1; j < rank; ++j) w = __fma_rn(-S.L[j][i], S.z[j], w);
      w = one_div(w, S.L[i][i]);
      __syncwarp();
      if (lane == 0) S.z[i] = w;
      __syncwarp();
    }
    if (lane < rank) S.coef[pl] = S.coef[pl] + S.z[lane];
    __syncwarp();
    if (pass == 0 && lane < rank) {
      double w = S.b[pl];
#pragma unroll 1
      for (int j = 0; j < k; ++j) w = __fma_rn(-S.G[pl][j], S.coef[j], w);
      rhs = w;
    }
  }
  const uint32_t flags = rank < k ? RRG_F_RANK_DEFICIENT : 0u;
  // Decisions the FP64 path must take itself: a rank cut (the reference's
  // rule works at eps^2 of the column norms), ill-conditioning, and
  // coefficients inside the ambiguity band of the drop (|c| < 1e-12) and
  // snap (|c - 1| < 1e-12) rules of the rebuilt tree.
  int why = -1;
  if (rank < k && a.certify) why = FB_RANK;
  else if (rank == k && min_ratio < a.fallback_tol) why = FB_ILL_COND;
  const double ci = lane < k ? S.coef[lane] : 0.0;
  const double fe = lane < m ? ferr(lane) : 0.0;
  const double ryy = one_sqrt(yy);
  if (why < 0 && a.certify) {
    // Coefficient error of the Gram solve: with relative errors u of the
    // Gram entries (the sums, kU, and the table's evaluation, ferr / rms of
    // each column) and the smallest relative pivot as the scaled
    // conditioning,
    //   |dc_i| <= u (|y| + sum_j |c_j| |f_j|) sqrt(k) / (lam |f_i|),  lam = min_ratio / k.
    // The drop (|c| < 1e-12) and snap (|c - 1| < 1e-12) rules of the rebuilt
    // tree are left to the FP64 path when c lies within 8 |dc_i| of them.
    double M = ryy;
#pragma unroll 1
    for (int i = 0; i < k; ++i) M = __fma_rn(fabs(S.coef[i]), S.root[i], M);
    double u = lane < m ? fmax(kU, one_div(fe, fmax((double)pr.rms[lane], 1e-300))) : kU;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) u = fmax(u, __shfl_xor_sync(0xffffffffu, u, o));
    const double lam = one_div(fmax(min_ratio, 1e-300), (double)k);
    bool snap = false, drop = false;
    if (lane < k) {
      const double dc = one_div(8.0 * u * M * one_sqrt((double)k), lam * fmax(S.root[lane], 1e-300));
      snap = lane < m && !(fabs(fabs(ci - 1.0) - kEps12) > dc);
      drop = !snap && !(fabs(fabs(ci) - kEps12) > dc);
    }
    const uint32_t sm = __ballot_sync(0xffffffffu, snap), any = sm | __ballot_sync(0xffffffffu, drop);
    if (any) why = (sm >> (__ffs(any) - 1)) & 1u ? FB_SNAP : FB_DROP;
  }
  const int kind = fabs(ci) < kEps12 ? 0 : (lane == m ? 1 : (fabs(ci - 1) < kEps12 ? 2 : 3));
  const double ceff = kind == 0 ? 0.0 : (kind == 2 ? 1.0 : ci);
  if (lane < k) {
    MixedTerm& tm = a.terms[c];
    out[lane] = ci;
    tm.hi[lane] = (float)ci;
    tm.lo[lane] = (float)(ci - (double)(float)ci);
    tm.kind[lane] = (int8_t)kind;
    S.z[lane] = ceff;
  }
  __syncwarp();
  // mag bounds the sums of |terms| behind every entry used (Cauchy-Schwarz:
  // sum |f_i f_j| <= sqrt(G_ii G_jj), sum |f_i y| <= sqrt(G_ii y'y))
  for (int e = lane; e < k * k; e += 32) {
    const double cc = S.z[e / k] * S.z[e % k];
    S.t[0][e] = cc;
    S.t[1][e] = fabs(cc) * S.root[e / k];
  }
  __syncwarp();
  if (lane > 1) return;
  // lane 0: y'y - 2 c'b + c'Gc; lane 1: mag
  double lin = 0.0, quad = 0.0, mag = yy;
#pragma unroll 1
  for (int i = 0; i < k; ++i) {
    if (lane == 0) {
      lin = __fma_rn(S.z[i], S.b[i], lin);
#pragma unroll 1
      for (int j = 0; j < k; ++j) quad = __fma_rn(S.t[0][i * k + j], S.G[i][j], quad);
    } else {
      mag = __fma_rn(2.0 * fabs(S.z[i]) * S.root[i], ryy, mag);
#pragma unroll 1
      for (int j = 0; j < k; ++j) mag = __fma_rn(S.t[1][i * k + j], S.root[j], mag);
    }
  }
  mag = __shfl_sync(0x3u, mag, 1);
  double err = 0.0;  // per-row error of the rebuilt sum
#pragma unroll 1
  for (int i = 0; i < m; ++i) err = __fma_rn(fabs(S.z[i]), ferr(i), err);
  if (lane != 0) return;
  double sse = yy - 2.0 * lin + quad;
  uint8_t p2 = 0;
  if (why < 0 && !(sse > 0.0 && kU * mag <= a.pass2_tol * sse)) {
    // the residual pass gives the SSE; certified rounds check it after
    p2 = 1;
    if (a.certify) a.cert_e[c] = err;
  } else if (why < 0 && a.certify && cert_bound(sse, err) > a.cert_tol) {
    why = FB_CERT;
  }
  if (why >= 0) {
    queue_fallback(why);
    p2 = 0;
    sse = -1.0;
  } else if (p2) {
    sse = -1.0;
  }
  a.sse1[c] = sse;
  a.pass2[c] = p2;
  a.res[c].rank = rank;
  a.res[c].flags |= flags;
}


// One block per distinct factor: both interpreters on kProbeRows rows spread
// evenly over the dataset (every row when n <= kProbeRows).  The squares are
// added by one warp, lane l taking the probed rows l, l + 32, ... in order.
// Bound by latency in small rounds and by the FP64 and integer pipes in large
// ones.  A warp for each factor, four factors a block, left most of the GPU idle
// in the first and mixed four programs' instructions in the second: 680 factors
// 0.45 ms with the solve, now 0.14 (256 threads 0.15, 128 threads 0.18); 8192
// random trees 10.0 ms, now 4.1; eight rounds at 1M rows 5.8 ms, now 2.4.
__global__ void __launch_bounds__(kProbeThreads) fac_probe_kernel(const uint32_t* code, const int2* meta,
                                                                  const double* K64, const float* K32,
                                                                  const float* K32lo, DevData ds, FacProbe* out,
                                                                  const int32_t* omap) {
  __shared__ double val[kProbeRows];
  __shared__ float dev_s;
  __shared__ uint32_t flags_s, cnt_s;
  const int f = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
  if (tid == 0) {
    dev_s = 0.f;
    flags_s = cnt_s = 0;
  }
  __syncthreads();
  const int2 mt = meta[f];
  const uint32_t* fc = code + mt.x;
  const int P = ds.n < kProbeRows ? (int)ds.n : kProbeRows;
  float dev = 0.f;
  uint32_t flags = 0, cnt = 0;
  for (int p = tid; p < P; p += kProbeThreads) {
    const int64_t row = ds.n < kProbeRows ? p : ((2 * (int64_t)p + 1) * ds.n) / (2 * kProbeRows);
    double f64[1] = {0.0};
    dfl fd = dfl_make(0.f, 0.f);
    val[p] = 0.0;  // adds nothing
    if (!probe_eval64<1>(fc, mt.y, K64, ds, row, f64) || !eval_row_df(fc, mt.y, K32, K32lo, ds, row, fd)) {
      flags |= FP_FAIL;
      continue;
    }
    const double v = f64[0];
    const bool n64 = v != v, i64 = !n64 && fabs(v) > DBL_MAX;
    const bool n32 = fd.hi != fd.hi, i32 = !n32 && fabsf(fd.hi) > FLT_MAX;
    if (n64) flags |= FP_NAN64;
    if (i64) flags |= FP_INF64;
    if (n64 != n32 || (i32 && !i64) || (i64 && !i32)) flags |= FP_BAD32;
    if (!n64 && !i64 && !n32 && !i32) {
      dev = fmaxf(dev, (float)fabs(dfl_to_double(fd) - v));
      val[p] = v;
      cnt += 1;
    }
  }
  flags = __reduce_or_sync(0xffffffffu, flags);
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  // deviations are not negative (or NaN, which fmaxf passes over): their bits order as integers
  const uint32_t d = __reduce_max_sync(0xffffffffu, __float_as_uint(dev));
  if (lane == 0) {
    atomicOr(&flags_s, flags);
    atomicAdd(&cnt_s, cnt);
    atomicMax(reinterpret_cast<uint32_t*>(&dev_s), d);
  }
  __syncthreads();
  if (tid >= 32) return;
  double ss = 0.0;
  for (int p = lane; p < P; p += 32) ss = __fma_rn(val[p], val[p], ss);
  ss = warp_sum(ss);
  if (lane == 0) {
    FacProbe r;
    r.dev = dev_s;
    r.rms = cnt_s > 0 ? (float)sqrt(ss / (double)cnt_s) : 0.f;
    r.flags = flags_s | (P == ds.n ? FP_ALL_ROWS : 0u);
    out[omap ? omap[f] : f] = r;
  }
}

// One thread per mixed candidate: its probe record and first NaN row from
// those of its factors.
__global__ void cand_probe_kernel(const rrg_cand* cands, const int32_t* list, int32_t n_list,
                                  const int32_t* cand_fac, const int32_t* fcol, const FacProbe* fp,
                                  const unsigned long long* fnan, ProbeOut* out, int64_t* nanrow) {
  const int li = blockIdx.x * blockDim.x + threadIdx.x;
  if (li >= n_list) return;
  const int c = list[li];
  const rrg_cand cd = cands[c];
  const int m = cd.mode == RRG_TUNED ? cd.n_factors : 1;
  ProbeOut r;
  r.nan64 = r.inf64 = r.bad32 = 0;
  r.all_rows = 0;
  unsigned long long first = 0x7f7f7f7f7f7f7f7full;
  for (int i = 0; i < kMixedMaxM; ++i) {
    r.dev[i] = 0.f;
    r.rms[i] = 0.f;
    if (i >= m) continue;
    const int f = cand_fac[(size_t)li * kMixedMaxM + i];
    const FacProbe p = fp[f];
    r.dev[i] = p.dev;
    r.rms[i] = p.rms;
    if (p.flags & FP_NAN64) r.nan64 |= 1u << i;
    if (p.flags & FP_INF64) r.inf64 |= 1u << i;
    if (p.flags & FP_BAD32) r.bad32 |= 1u << i;
    if (p.flags & FP_FAIL) r.bad32 = 0xffffffffu;
    if (p.flags & FP_ALL_ROWS) r.all_rows = 1u;
    const unsigned long long fr = fnan[fcol ? fcol[f] : f];
    first = fr < first ? fr : first;
  }
  out[c] = r;
  nanrow[c] = (int64_t)first;
}

// One thread per candidate of the residual pass of a certified round: the
// bound of cert_fitness_bound on its residual-pass SSE (partials summed in
// the order of finalize_kernel); above the tolerance it is queued for FP64.
__global__ void cert_resid_kernel(const int32_t* mlist, const int32_t* list2, int32_t n2, const double* sse_part,
                                  int nb, const double* cert_e, DevData ds, double cert_tol, int32_t* fallback,
                                  int32_t fallback_cap, uint32_t* reasons, const int32_t* n2_dev) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n2 || (n2_dev && i >= *n2_dev)) return;
  const int c = mlist[list2[i]];
  const double E = cert_e[c];
  if (!(E >= 0.0)) return;
  double sse = 0.0;
  for (int j = 0; j < nb; ++j) sse = __dadd_rn(sse, sse_part[(int64_t)c * nb + j]);
  if (cert_fitness_bound(sse, E, (double)ds.n, ds.sst) > cert_tol) {
    const int slot = atomicAdd(fallback, 1);
    if (slot < fallback_cap) fallback[1 + slot] = c;
    atomicAdd(reasons + FB_CERT, 1u);
  }
}

__global__ void to_f32_kernel(const double* src, float* dst, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    dst[i] = (float)src[i];
}
__global__ void split_f32_kernel(const double* src, float* hi, float* lo, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const dfl v = dfl_from_double(src[i]);
    hi[i] = v.hi;
    lo[i] = v.lo;
  }
}

// ----------------------------------------------------------- launchers ----
bool launch_fac_probe(const uint32_t* code, const int2* meta, int32_t nf, const double* K64, const float* K32,
                      const float* K32lo, const DevData& ds, FacProbe* out, cudaStream_t st, const int32_t* omap) {
  if (nf <= 0) return true;
  fac_probe_kernel<<<nf, kProbeThreads, 0, st>>>(code, meta, K64, K32, K32lo, ds, out, omap);
  return launch_ok("launch_fac_probe");
}
bool launch_cand_probe(const rrg_cand* cands, const int32_t* list, int32_t n_list, const int32_t* cand_fac,
                       const int32_t* fcol, const FacProbe* fp, const unsigned long long* fnan, ProbeOut* out,
                       int64_t* nanrow, cudaStream_t st) {
  if (n_list <= 0) return true;
  cand_probe_kernel<<<(n_list + 127) / 128, 128, 0, st>>>(cands, list, n_list, cand_fac, fcol, fp, fnan, out,
                                                          nanrow);
  return launch_ok("launch_cand_probe");
}
bool launch_cert_resid(const int32_t* mlist, const int32_t* list2, int32_t n2, const double* sse_part, int nb,
                       const double* cert_e, const DevData& ds, double cert_tol, int32_t* fallback,
                       int32_t fallback_cap, uint32_t* reasons, cudaStream_t st, const int32_t* n2_dev) {
  if (n2 <= 0) return true;
  cert_resid_kernel<<<(n2 + 127) / 128, 128, 0, st>>>(mlist, list2, n2, sse_part, nb, cert_e, ds, cert_tol, fallback,
                                                      fallback_cap, reasons, n2_dev);
  return launch_ok("launch_cert_resid");
}
bool launch_solve(const SolveArgs& a, cudaStream_t st) {
  if (a.n_list <= 0) return true;
  mixed_solve_kernel<<<(a.n_list + 3) / 4, 128, 0, st>>>(a);
  return launch_ok("launch_solve");
}
bool launch_to_f32(const double* src, float* dst, int64_t n, cudaStream_t st) {
  to_f32_kernel<<<1024, 256, 0, st>>>(src, dst, n);
  return launch_ok("launch_to_f32");
}
bool launch_split_f32(const double* src, float* hi, float* lo, int64_t n, cudaStream_t st) {
  split_f32_kernel<<<1024, 256, 0, st>>>(src, hi, lo, n);
  return launch_ok("launch_split_f32");
}

}  // namespace rrd
