// Plain FP64 fitness path: the drop-in form of tune_constants + fitness
// (rils_rols_cpp/rils_rols_cpp.cpp:445-541).
//
//   plain_eval   evaluates every factor program of a candidate on every row
//                (node::evaluate_all, node.cpp:5-95) into the A arena;
//   (the column-pivoted QR on [A | 1 | y] is in qr_small.cu, one block per
//                candidate, and in qr_chunk.cu, over the GPU)
//   plain_resid  the rebuilt sum  sum_i c_i * f_i  with the drop / snap rules
//                of rils_rols_cpp.cpp:488-517 and its squared residual;
//   finalize     R2, RMSE and the NaN sentinel (rils_rols_cpp.cpp:40-49, 520-541).
#include <algorithm>
#include <cfloat>
#include <cstdint>

#include "../common/rr_math_split.h"
#include "../common/rr_sum.h"
#include "common.cuh"
#include "plain.cuh"
#include "qr_ops.cuh"
#include "reduce.cuh"

namespace rrd {

namespace {

constexpr int kMaxK = RRG_MAX_TERMS;

// Operators of the FP64 interpreter.  Sums take the FP64 pipe, one instruction
// each; products, quotients, roots and comparisons are formed on the integer
// pipes (csrc/common/fp64_int.h) and the elementary functions in their split
// forms (rr_math_split.h): the kernel is bound by the FP64 pipe (an
// instruction holds it for 16 cycles), so what leaves it is what is saved.
// GB300, the FP64 evaluation of a 660-candidate local-search round at 1M rows with
// native operations / with these, all else alike: 23.2 / 17.4 ms (12.8 with the
// pieces of eval_pieces and shared memory by need).  The results are the same bits.
__device__ __forceinline__ double bin64(int base, double a, double b) {
  switch (base) {
    case RRG_ADD: return __dadd_rn(a, b);
    case RRG_SUB: return __dsub_rn(a, b);
    case RRG_MUL: return fi_mul(a, b);
    case RRG_DIV: return fi_div(a, b);
    case RRG_POW: return rr_pow(a, b);
    case RRG_LT: return fi_lt(a, b) ? 1.0 : 0.0;
    case RRG_EQ: return fi_eq(a, b) ? 1.0 : 0.0;
    case RRG_NE: return fi_eq(a, b) ? 0.0 : 1.0;
    case RRG_MIN: return fi_lt(a, b) ? a : b;
    case RRG_MAX: return fi_lt(b, a) ? a : b;
    default: return __longlong_as_double(0x7ff8000000000000ll);
  }
}

// Runs the code of one candidate on `row`; factor slot s is written to
// out[s * n_pad + row], or, with ONE (a one-column program), returned instead.
// Spill stack in shared memory, stride blockDim.x.  Table programs also read
// columns of T (same rows, column stride n_pad).
template <bool ONE>
__device__ __forceinline__ double run_row64(const uint32_t* code, int len, const double* consts, const DevData& ds,
                                            int64_t row, double* st, int levels, double* out, const double* T,
                                            uint32_t* status) {
  double tos = 0.0;
  int sp = 0;
  const int stride = blockDim.x;
  for (int pc = 0; pc < len; ++pc) {
    const uint32_t w = code[pc];
    const int op = (int)(w & 0xffu);
    const uint32_t arg = w >> 8;
    switch (op) {
      case RRG_OP_LDV: tos = ds.X64[(int64_t)arg * ds.n_pad + row]; break;
      case RRG_OP_LDC: tos = consts[arg]; break;
      case RRG_OP_PSV:
        if (sp >= levels) { atomicOr(status, ST_STACK); return tos; }
        st[sp++ * stride] = tos;
        tos = ds.X64[(int64_t)arg * ds.n_pad + row];
        break;
      case RRG_OP_PSC:
        if (sp >= levels) { atomicOr(status, ST_STACK); return tos; }
        st[sp++ * stride] = tos;
        tos = consts[arg];
        break;
      case RRG_OP_SIN:
      case RRG_OP_COS: tos = rrs_sincos(tos, op - RRG_OP_SIN); break;
      case RRG_OP_LN: tos = rrs_log(tos); break;
      case RRG_OP_EXP: tos = rrs_exp(tos); break;
      case RRG_OP_SQRT: tos = fi_sqrt(tos); break;
      case RRG_OP_SQR: tos = fi_mul(tos, tos); break;
      case kOpLDT: tos = T[(int64_t)arg * ds.n_pad + row]; break;
      case kOpPST:
        if (sp >= levels) { atomicOr(status, ST_STACK); return tos; }
        st[sp++ * stride] = tos;
        tos = T[(int64_t)arg * ds.n_pad + row];
        break;
      case RRG_OP_EMIT:
        if (!ONE) out[(int64_t)arg * ds.n_pad + row] = tos;
        sp = 0;
        break;
      default: {
        const int kk = op - RRG_OP_BIN;
        if (kk < 0 || kk >= 8 * RRG_N_BASE) { atomicOr(status, ST_BAD_CODE); return tos; }
        const int base = kk >> 3, src = (kk & 7) >> 1, dir = kk & 1;
        double other;
        if (src == RRG_SRC_S) {
          if (sp <= 0) { atomicOr(status, ST_STACK); return tos; }
          other = st[--sp * stride];
        } else if (src == RRG_SRC_V) {
          other = ds.X64[(int64_t)arg * ds.n_pad + row];
        } else if (src == kSrcT) {
          other = T[(int64_t)arg * ds.n_pad + row];
        } else {
          other = consts[arg];
        }
        tos = dir == RRG_DIR_N ? bin64(base, other, tos) : bin64(base, tos, other);
      }
    }
  }
  return tos;
}

// One-column table program on rows [r0, r1) of this block, written to Ac;
// the column's flags (NaN, infinite or overflowing square, non-trivial tail)
// merged into *cs.  stop: a column that no program reads as an operand; once
// some block has stored a NaN at row kStopRow or later, the blocks leave off
// (the block of row 0 after its first rows, so that rows below kStopRow are
// all there).  2048 random trees at 100k rows, seven of eight with a NaN
// somewhere: with the pieces (eval_pieces) and the shared columns left out that no
// factor needs (eval_two_parts) 6.9 ms, where all their rows took 78.5.
__device__ __forceinline__ void eval_column_stats(const uint32_t* code, int len, const double* consts,
                                                  const DevData& ds, int64_t r0, int64_t r1, double* st, int levels, double* Ac,
                                                  const double* T, uint32_t* status, ColStat* cs, bool stop,
                                                  volatile int* found) {
  static_assert(kStopRow <= 256, "within the first rows of a block");
  uint32_t f = 0;
  const bool skip = stop && (__ldcg(&cs->flags) & kCsStop) != 0;  // (any mix of answers in a block does)
  for (int64_t r = r0 + threadIdx.x; r < r1; r += blockDim.x) {
    if (stop && r >= blockDim.x && (skip || (r - r0 >= blockDim.x && *found))) break;
    const double v = run_row64<true>(code, len, consts, ds, r, st, levels, nullptr, T, status);
    Ac[r] = v;
    // on the bits of |v| (non-negative doubles order as integers, NaN above)
    const unsigned long long a = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
    if (a > 0x7ff0000000000000ull) {
      f |= kCsNaN;
      if (stop && r >= kStopRow && !*found) {
        *found = 1;
        atomicOr(&cs->flags, kCsStop | kCsNaN | kCsTail);
      }
    } else if (a > 0x5ff01c2a01d98729ull) {
      f |= kCsBig;  // above 1.35e154: infinite, or its square overflows
    }
    if (r >= 1 && a > 0x20ca2fe76a3f9475ull) f |= kCsTail;  // above 1e-150, or not finite
  }
  f = __reduce_or_sync(0xffffffffu, f);
  if ((threadIdx.x & 31) == 0 && f) atomicOr(&cs->flags, f);
}

}  // namespace

// ------------------------------------------------------------- kernels ----
__global__ void __launch_bounds__(256) table_eval_list_kernel(DevBatch b, DevData ds, const PlainCand* pc,
                                                               const int32_t* cols, const int32_t* count,
                                                               int min_nbc, int max_nbc, double* A, uint32_t* status,
                                                               ColStat* cst, EvalRows rows) {
  extern __shared__ double smem[];
  const int cnt = *count;
  if (cnt <= 0) return;
  const int nbc = max(min_nbc, min(max_nbc, (int)((gridDim.x + cnt - 1) / cnt)));
  const int64_t items = (int64_t)cnt * nbc;
  double* st = smem + threadIdx.x;
  uint32_t* code_s = reinterpret_cast<uint32_t*>(smem + rows.levels * blockDim.x);
  for (int64_t w = blockIdx.x; w < items; w += gridDim.x) {
    const int c = cols[w % cnt];
    const int bi = (int)(w / cnt);
    if (rows.live && !rows.live[pc[c].a_col]) continue;  // uniform
    const rrg_cand cd = b.cands[c];
    const int64_t nr = rows.hi - rows.lo;
    const int64_t r0 = rows.lo + nr * bi / nbc, r1 = rows.lo + nr * (bi + 1) / nbc;
    const bool staged = cd.code_len < rows.words;
    volatile int* found = reinterpret_cast<int*>(code_s + rows.words - 1);
    __syncthreads();  // the previous item's program is no longer read
    if (threadIdx.x == 0) *found = 0;
    if (staged)
      for (int i = threadIdx.x; i < cd.code_len; i += blockDim.x) code_s[i] = b.code[cd.code_offset + i];
    __syncthreads();
    const uint32_t* code = staged ? code_s : b.code + cd.code_offset;
    eval_column_stats(code, cd.code_len, b.consts, ds, r0, r1, st, rows.levels, A + pc[c].a_col * ds.n_pad, A, status,
                      &cst[pc[c].a_col], cd.reserved == kColStop, found);
  }
}

// grid (candidates, nb): nb pieces of the rows [rows.lo, rows.hi).  Candidates first, so
// that a piece's NaN is known before most blocks of the later pieces start.
__global__ void __launch_bounds__(256) plain_eval_kernel(DevBatch b, DevData ds, const PlainCand* pc,
                                                          const int32_t* list, int cand0, double* A, uint32_t* status,
                                                          ColStat* cst, EvalRows rows) {
  extern __shared__ double smem[];
  after_previous();
  const int c = list ? list[cand0 + blockIdx.x] : cand0 + blockIdx.x;
  const rrg_cand cd = b.cands[c];
  if (rows.live && !rows.live[pc[c].a_col]) return;
  const int nb = gridDim.y;
  const int64_t nr = rows.hi - rows.lo;
  const int64_t r0 = rows.lo + nr * blockIdx.y / nb, r1 = rows.lo + nr * (blockIdx.y + 1) / nb;
  double* st = smem + threadIdx.x;  // spill stack, rows.levels * blockDim.x doubles
  uint32_t* code_s = reinterpret_cast<uint32_t*>(smem + rows.levels * blockDim.x);
  const bool staged = cd.code_len < rows.words;
  volatile int* found = reinterpret_cast<int*>(code_s + rows.words - 1);
  if (threadIdx.x == 0) *found = 0;
  if (staged)
    for (int i = threadIdx.x; i < cd.code_len; i += blockDim.x) code_s[i] = b.code[cd.code_offset + i];
  __syncthreads();
  const uint32_t* code = staged ? code_s : b.code + cd.code_offset;
  double* Ac = A + pc[c].a_col * ds.n_pad;
  if (cst) {
    eval_column_stats(code, cd.code_len, b.consts, ds, r0, r1, st, rows.levels, Ac, A, status, &cst[pc[c].a_col],
                      cd.reserved == kColStop, found);
    return;
  }
  for (int64_t r = r0 + threadIdx.x; r < r1; r += blockDim.x)
    run_row64<false>(code, cd.code_len, b.consts, ds, r, st, rows.levels, Ac, A, status);
}

// One block.  The columns that still count after some rows are evaluated: the
// factors without a NaN that settles them, the operands kept as factors, and
// what these read, level by level (latency; some 20 us for 4600 columns in 15
// levels, against milliseconds of evaluation that it saves).
__global__ void __launch_bounds__(1024) live_columns_kernel(LiveArgs a) {
  auto slot_of = [&](int e) { return a.wcol ? a.wcol[e] : e; };
  const int tid = threadIdx.x, ne = a.level_end[a.n_levels - 1];
  for (int e = tid; e < ne; e += blockDim.x) {
    const int s = slot_of(e);
    bool v = a.kind[e] != kColShared && !(a.only && a.only[e] != a.only_value);
    if (v && a.kind[e] == kColStop)
      v = a.cst ? !(a.cst[s].flags & kCsStop) : a.fnan[s] >= (unsigned long long)a.rows;
    a.live[s] = v ? 1 : 0;
  }
  __syncthreads();
  for (int L = a.n_levels - 1; L > 0; --L) {
    for (int e = a.level_end[L - 1] + tid; e < a.level_end[L]; e += blockDim.x) {
      if (!a.live[slot_of(e)]) continue;
      const int2 m = a.meta[e];
      for (int i = 0; i < m.y; ++i) {
        const uint32_t w = a.code[m.x + i];
        const int op = (int)(w & 0xffu);
        if (op == kOpLDT || op == kOpPST || (op >= RRG_OP_BIN && (((op - RRG_OP_BIN) & 7) >> 1) == kSrcT))
          a.live[w >> 8] = 1;
      }
    }
    __syncthreads();
  }
}
bool launch_live_columns(const LiveArgs& a, cudaStream_t st) {
  if (a.n_levels <= 0) return true;
  live_columns_kernel<<<1, 1024, 0, st>>>(a);
  return launch_ok("launch_live_columns");
}

int plain_qr_bucket(int cols) { return cols <= 4 ? 4 : (cols <= 8 ? 8 : (cols <= 16 ? 16 : kMaxK + 1)); }

// SSE of the rebuilt sum per (candidate, chunk of RR_CHUNK rows) item in the
// fixed order of csrc/common/rr_sum.h; the grid walks the items.
//
// Bound: the FP64 pipe.  The scaled terms' products and the squared residual
// are formed on the integer pipes (csrc/common/fp64_int.h), so a row of m scaled
// terms and a free term takes m + 2 FP64 additions (2 m + 4 FP64 instructions
// before); kResidRows rows of a lane are handled together, term by term, so that
// their loads are in flight at once.  GB300, 605 candidates at 1M rows: 10.3 ms
// before, 6.4 now.
// SEG = 4: blocks of 1024 threads, four to a lane, each forming a quarter of
// the lane's squares before the lane's sum passes from one to the next: for
// launches that leave most SMs without a block (one candidate at 1M rows has
// 62 chunks: 0.125 ms before, 0.045 now).
constexpr int kResidRows = 8;
template <int SEG>
__global__ void __launch_bounds__(256 * SEG, 4 / SEG) plain_resid_kernel(DevBatch b, DevData ds, const PlainCand* pc,
                                                                const int32_t* list, int cand0, int n_cand,
                                                                const double* A, const double* coefs, double* partial,
                                                                const int32_t* colmap, const int32_t* dcount) {
  after_previous();
  __shared__ double red[8], lane_acc[256];
  __shared__ fi_factor cs[kMaxK];
  __shared__ int kind[kMaxK];  // 0 skip, 1 free term, 2 bare factor, 3 scaled factor
  __shared__ const double* colp[kMaxK];
  constexpr int kSegRows = RR_CHUNK / 256 / SEG;  // rows of a lane per thread
  static_assert(kSegRows % kResidRows == 0, "whole row groups");
  const int lane = threadIdx.x & 255, seg = threadIdx.x >> 8;
  const int nb = (int)((ds.n + RR_CHUNK - 1) / RR_CHUNK);
  const int cnt = dcount ? min(max(*dcount - cand0, 0), n_cand) : n_cand;
  const int64_t items = (int64_t)cnt * nb;
  for (int64_t it = blockIdx.x; it < items; it += gridDim.x) {
    const int i = (int)(it / nb), ch = (int)(it % nb);
    const int c = list ? list[cand0 + i] : cand0 + i;
    const rrg_cand cd = b.cands[c];
    const bool tuned = cd.mode == RRG_TUNED;
    if (tuned && (pc[c].pad & 1)) {
      // all-NaN coefficients: every row's rebuilt sum is NaN
      if (threadIdx.x == 0)
        partial[(int64_t)c * nb + ch] = ch == 0 ? __longlong_as_double(0x7ff8000000000000ll) : 0.0;
      continue;
    }
    const int k = tuned ? pc[c].k : 1;
    const int m = tuned ? k - 1 : 1;
    __syncthreads();  // the previous item's terms are no longer read
    for (int t = threadIdx.x; t < k; t += blockDim.x) {
      const double ci = tuned ? coefs[cd.coef_offset + t] : 1.0;
      cs[t] = fi_factor_of(ci);
      kind[t] = fabs(ci) < kEps12 ? 0 : (tuned && t == m ? 1 : (fabs(ci - 1) < kEps12 ? 2 : 3));
      if (t < m) colp[t] = factor_column(A, ds.n_pad, pc[c].a_col, t, colmap);
    }
    __syncthreads();
    const int64_t r0 = (int64_t)ch * RR_CHUNK;
    const int64_t first = r0 + lane + (int64_t)seg * kSegRows * 256;
    double acc = 0.0, sq[SEG == 1 ? kResidRows : kSegRows];
#pragma unroll 1
    for (int u0 = 0; u0 < kSegRows; u0 += kResidRows) {
      const int64_t i0 = first + 256 * u0;
      if (i0 >= ds.n) break;
      const bool full = i0 + 256 * (kResidRows - 1) < ds.n;
      if (SEG == 1 && !full) {
        // the last rows one at a time (small datasets have few to a lane)
        for (int64_t r = i0; r < ds.n; r += 256) {
          double yp = 0.0;
          bool have = false;
          for (int t = 0; t < k; ++t) {
            const int kd = kind[t];
            if (kd == 0) continue;
            const double v = kd == 1 ? 1.0 : __ldg(colp[t] + r);
            const double term = kd == 1 ? cs[t].b : (kd == 2 ? v : fi_mul_by(v, cs[t]));
            yp = have ? __dadd_rn(yp, term) : term;
            have = true;
          }
          const double e = __dsub_rn(__ldg(ds.y64 + r), yp);
          acc = __dadd_rn(acc, fi_mul(e, e));
        }
        break;
      }
      double yp[kResidRows], e[kResidRows];
      bool have = false;
      for (int t = 0; t < k; ++t) {
        const int kd = kind[t];
        if (kd == 0) continue;
        const fi_factor f = cs[t];
        if (kd == 1) {
#pragma unroll
          for (int u = 0; u < kResidRows; ++u) yp[u] = have ? __dadd_rn(yp[u], f.b) : f.b;
        } else {
          const double* col = colp[t];
          double v[kResidRows];
#pragma unroll
          for (int u = 0; u < kResidRows; ++u)
            v[u] = SEG == 1 || full || i0 + 256 * u < ds.n ? __ldg(col + i0 + 256 * u) : 0.0;
#pragma unroll
          for (int u = 0; u < kResidRows; ++u) {
            const double term = kd == 2 ? v[u] : fi_mul_by(v[u], f);
            yp[u] = have ? __dadd_rn(yp[u], term) : term;
          }
        }
        have = true;
      }
#pragma unroll
      for (int u = 0; u < kResidRows; ++u) {
        const double y = SEG == 1 || full || i0 + 256 * u < ds.n ? __ldg(ds.y64 + i0 + 256 * u) : 0.0;
        e[u] = __dsub_rn(y, have ? yp[u] : 0.0);
        e[u] = fi_mul(e[u], e[u]);
      }
      if constexpr (SEG == 1) {
#pragma unroll
        for (int u = 0; u < kResidRows; ++u) acc = __dadd_rn(acc, e[u]);
      } else {
        // (constant indexes keep the squares in registers)
#pragma unroll
        for (int g = 0; g < kSegRows; g += kResidRows)
          if (g == u0) {
#pragma unroll
            for (int u = 0; u < kResidRows; ++u) sq[g + u] = e[u];
          }
      }
    }
    if constexpr (SEG > 1) {
      // the lane's sum in row order: each quarter goes on from the one before
      for (int s = 0; s < SEG; ++s) {
        if (seg == s) {
          acc = s ? lane_acc[lane] : 0.0;
#pragma unroll
          for (int u = 0; u < kSegRows; ++u)
            if (first + 256 * u < ds.n) acc = __dadd_rn(acc, sq[u]);
          lane_acc[lane] = acc;
        }
        __syncthreads();
      }
      acc = lane_acc[lane];
    }
    // the first 256 threads fold the lanes
    const double ws = warp_sum(acc);
    if (seg == 0 && (lane & 31) == 0) red[lane >> 5] = ws;
    __syncthreads();
    if (threadIdx.x == 0) {
      double s = 0.0;
      for (int w = 0; w < 8; ++w) s = __dadd_rn(s, red[w]);
      partial[(int64_t)c * nb + ch] = s;
    }
  }
}

bool launch_plain_resid(DevBatch b, const DevData& ds, const PlainCand* pc, const int32_t* list, int cand0, int n_cand,
                        const double* A, const double* coefs, double* partial, const int32_t* colmap,
                        const int32_t* dcount, int sm_count, cudaStream_t st, bool chained) {
  if (n_cand <= 0) return true;
  const int64_t items = (int64_t)n_cand * ((ds.n + RR_CHUNK - 1) / RR_CHUNK);
  // four threads a lane while that gives every SM at most two such blocks and
  // a lane has more rows than one thread takes together
  if (!dcount && items <= 2 * sm_count && ds.n > 256 * kResidRows)
    plain_resid_kernel<4><<<(int)items, 1024, 0, st>>>(b, ds, pc, list, cand0, n_cand, A, coefs, partial, colmap,
                                                       dcount);
  else
    launch_next(chained, plain_resid_kernel<1>, dim3((unsigned)std::min<int64_t>(items, 16 * (int64_t)sm_count)), 256,
                0, st, b, ds, pc, list, cand0, n_cand, A, coefs, partial, colmap, dcount);
  return launch_ok("residual");
}

// one thread per candidate: R2, RMSE, sentinel, rebuilt size
__global__ void finalize_kernel(DevBatch b, DevData ds, const int32_t* list, int cand0, int cand1,
                                const double* partial, int nb, const double* coefs, rrg_result* res,
                                uint32_t flags_or, const double* sse_direct, const int32_t* dcount) {
  after_previous();
  const int i = cand0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= cand1 || (dcount && i >= *dcount)) return;
  const int c = list ? list[i] : i;
  const rrg_cand cd = b.cands[c];
  double ssr = 0.0;
  if (sse_direct && !(sse_direct[c] < 0.0)) {
    ssr = sse_direct[c];
  } else {
    for (int j = 0; j < nb; ++j) ssr = __dadd_rn(ssr, partial[(int64_t)c * nb + j]);
  }
  const double r2 = __dsub_rn(1.0, __ddiv_rn(ssr, ds.sst));
  const double rmse = __dsqrt_rn(__ddiv_rn(ssr, (double)ds.n));
  rrg_result out = res[c];
  out.flags |= flags_or;
  int size = 0;
  if (cd.mode == RRG_TUNED) {
    const int m = cd.n_factors;
    int kept = 0;
    for (int i = 0; i <= m; ++i) {
      const double ci = coefs[cd.coef_offset + i];
      if (fabs(ci) < kEps12) continue;
      ++kept;
      if (i == m) size += 1;
      else if (fabs(ci - 1) < kEps12) size += b.factors[cd.first_factor + i].n_nodes;
      else size += 2 + b.factors[cd.first_factor + i].n_nodes;
    }
    size = kept == 0 ? 1 : size + kept - 1;
    out.n_coef = m + 1;
    if (out.rank < m + 1) out.flags |= RRG_F_RANK_DEFICIENT;
  } else {
    size = b.factors[cd.first_factor].n_nodes;
    out.n_coef = 0;
    out.rank = 0;
  }
  if (r2 != r2 || rmse != rmse) {
    out.loss = 1000;
    out.rmse = 1000;
    out.size = 1000;
    out.flags |= RRG_F_NONFINITE;
  } else {
    out.loss = __dsub_rn(1.0, r2);
    out.rmse = rmse;
    out.size = size;
  }
  res[c] = out;
}

// ----------------------------------------------------------- launchers ----
// Result records of the listed candidates back to zero before a re-scoring.
__global__ void clear_results_kernel(const int32_t* list, int n, rrg_result* res, const int32_t* dcount) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && !(dcount && i >= *dcount)) res[list[i]] = rrg_result{};
}

// Those, and the statistics of the columns about to be evaluated: one launch.
__global__ void table_begin_kernel(const int32_t* list, int n, rrg_result* res, const int32_t* slots, int n_slots,
                                   ColStat* cst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) res[list[i]] = rrg_result{};
  if (i < n_slots) cst[slots[i]] = ColStat{};
}
bool launch_table_begin(const int32_t* list, int n, rrg_result* res, const int32_t* slots, int n_slots, ColStat* cst,
                        cudaStream_t st) {
  const int m = n > n_slots ? n : n_slots;
  if (m <= 0) return true;
  table_begin_kernel<<<(m + 255) / 256, 256, 0, st>>>(list, n, res, slots, n_slots, cst);
  return launch_ok("table_begin");
}

// The outcome of the column-pivoted QR (ColPivHouseholderQR.h:482-608, as
// restated by the oracle) on [f_0 .. f_{m-1}, 1] when its first pivot has a
// non-finite norm.  Pivot selection keeps the first maximum under '>', so a
// NaN norm is chosen only when it heads the remaining columns and a +inf
// norm beats every finite one: the first pivot is non-finite when column 0's
// norm is NaN or some column's norm is +inf (an infinite value or an
// overflowing square, without NaN).  With a non-trivial tail in every column
// (some row after the first above 1e-150: the reflector is formed and every
// norm is non-zero), that pivot yields tau = NaN, which turns every other
// column and its norm NaN; no step cuts the rank (step 0 compares against an
// infinite or NaN threshold, later steps against NaN norms), so all
// coefficients are NaN at full rank.  A finite first pivot can leave a column
// with an exactly zero norm that a later step cuts, so NaN columns further
// on are left to the QR.
constexpr int kGramCols = 9;  // finite columns (the free term included) of the certificate below; wider: the QR
constexpr int kGramE = kGramCols * (kGramCols + 1) / 2;
// Returns the candidate's PlainCand::pad: 1 decided (written), 2 for nan_gram, else 0.
__device__ __forceinline__ int classify_candidate(const DevBatch& b, int c, const PlainCand& p, const int32_t* colmap,
                                                  const ColStat* cs, int64_t rows, double* coefs, rrg_result* res,
                                                  uint32_t* decided) {
  const rrg_cand cd = b.cands[c];
  const int k = p.k, m = k - 1;
  if (cd.mode != RRG_TUNED || m < 1 || rows < (int64_t)k + 2) return 0;
  bool tails = true, inf_norm = false, nan0 = false, any_nan = false;
  int nf = 0;
  for (int j = 0; j < m; ++j) {
    const uint32_t f = cs[colmap[p.a_col + j]].flags;
    if (!(f & kCsTail)) tails = false;
    if (f & kCsNaN) {
      any_nan = true;
      if (j == 0) nan0 = true;
    } else {
      ++nf;
      if (f & kCsBig) inf_norm = true;
    }
  }
  if (!tails) return 0;
  if (nan0 || inf_norm) {
    double* out = coefs + cd.coef_offset;
    for (int j = 0; j < k; ++j) out[j] = __longlong_as_double(0x7ff8000000000000ll);
    res[c].rank = k;
    atomicAdd(decided, 1u);
    return 1;
  }
  // a NaN column further right: left to nan_gram_* (bit 1), which decides it
  // when the finite columns are well conditioned
  return any_nan && nf + 1 <= kGramCols ? 2 : 0;
}

// A NaN column at position q >= 1, column 0 finite, no infinite norm, every
// tail non-trivial: step 0 pivots on a finite column (NaN norms never win the
// '>' scan unless they head the remaining columns) with tau != 0, which turns
// every NaN-holding column entirely NaN; NaN columns do not move before step
// q, where the first of them heads the remaining columns and is chosen; its
// tau is NaN and every later norm and coefficient NaN, so the result is
// all-NaN coefficients at full rank, unless some step before q cut the rank.
// Steps before q factor finite columns only, so no cut is possible when the
// finite columns (the free term included) are well conditioned: every pivot
// of their pivoted Cholesky above 1e-8 of its column's squared norm and
// 1e-24 of the largest (the reference cuts at eps^2 ~ 5e-32 of the largest,
// and a remaining norm that far above it cannot be rounded down to it).
// nan_gram_kernel forms their FP64 Gram matrix (a certificate: any summation
// order), nan_gram_decide_kernel factors it.
__device__ __forceinline__ int gram_finite_cols(const PlainCand& p, const int32_t* colmap, const ColStat* cs,
                                                const double* T, int64_t n_pad, const double* (&colp)[kGramCols]) {
  const int m = p.k - 1;
  int nf = 0;
  for (int j = 0; j < m && nf < kGramCols - 1; ++j) {
    const int32_t t = colmap[p.a_col + j];
    if (!(cs[t].flags & kCsNaN)) colp[nf++] = T + (int64_t)t * n_pad;
  }
  return nf;
}

// The Gram entries of the candidate's finite columns over `steps` runs of 256
// rows, run i from row_of(i) (rows at or beyond `end` are left out), by a block
// of 256 threads, into out.
template <class RowOf>
__device__ __forceinline__ void gram_block(const PlainCand& p, const int32_t* colmap, const ColStat* cs,
                                           const double* T, int64_t n_pad, int64_t steps, RowOf row_of, int64_t end,
                                           double (*red)[kGramE], double* out) {
  const double* colp[kGramCols];
  const int nf = gram_finite_cols(p, colmap, cs, T, n_pad, colp);
  const int K = nf + 1;  // the free term last
  double part[kGramE];
#pragma unroll
  for (int e = 0; e < kGramE; ++e) part[e] = 0.0;
  for (int64_t i = 0; i < steps; ++i) {
    const int64_t r = row_of(i) + threadIdx.x;
    if (r >= end) continue;
    double v[kGramCols];
#pragma unroll
    for (int a = 0; a < kGramCols; ++a) v[a] = a < nf ? colp[a][r] : 1.0;
    int e = 0;
#pragma unroll
    for (int a = 0; a < kGramCols; ++a)
#pragma unroll
      for (int bb = a; bb < kGramCols; ++bb, ++e)
        if (bb < K) part[e] = fma(v[a], v[bb], part[e]);
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  int e = 0;
#pragma unroll
  for (int a = 0; a < kGramCols; ++a)
#pragma unroll
    for (int bb = a; bb < kGramCols; ++bb, ++e) {
      const double t = bb < K ? warp_sum(part[e]) : 0.0;  // uniform
      if (l == 0) red[w][e] = t;
    }
  __syncthreads();
  for (int i = threadIdx.x; i < kGramE; i += blockDim.x) {
    double t = 0.0;
    for (int ww = 0; ww < 8; ++ww) t += red[ww][i];
    out[i] = t;
  }
}

__global__ void __launch_bounds__(256) nan_gram_kernel(const int32_t* list, int cnt, const PlainCand* pc,
                                                       const int32_t* colmap, const ColStat* cs, const double* T,
                                                       int64_t n, int64_t n_pad, double* gpart,
                                                       const int32_t* dcount) {
  __shared__ double red[8][kGramE];
  const int i = blockIdx.x;
  if (i >= cnt || (dcount && i >= *dcount)) return;
  const PlainCand p = pc[list[i]];
  if (!(p.pad & 2)) return;
  const int64_t r0 = n * (int64_t)blockIdx.y / gridDim.y, r1 = n * (int64_t)(blockIdx.y + 1) / gridDim.y;
  gram_block(p, colmap, cs, T, n_pad, (r1 - r0 + 255) / 256, [&](int64_t s) { return r0 + 256 * s; }, r1, red, gpart + ((int64_t)i * gridDim.y + blockIdx.y) * kGramE);
}

// Whether the certificate of nan_gram holds for candidate p (1; 0 not; -1 not,
// and a column all but depends on the others, as twice the same factor does),
// from the nbx partial Gram matrices at gp.  n > 0: they are those of some of the n rows, and
// the columns' squared norms are in cs; a Gram matrix over all rows is larger
// (in the order of semidefinite matrices), and so is what is left of a column
// after any other columns are taken out.  The QR may take the pivots in another
// order then.  What any order leaves of a column is at least the sample matrix's
// smallest eigenvalue, and pivoted elimination's smallest pivot is at most
// K 4^(K - 1) times that; so the pivots have to be that much above the bound of
// the all-rows form, 1e-24 of the largest squared norm, which then holds in the
// QR's order too: what is left of a column is at least 1e-12 of the largest norm
// and of its own, far above rounding (2^-53) and above the cut (2^-52).
__device__ __noinline__ int gram_certifies(const PlainCand& p, const int32_t* colmap, const ColStat* cs, int nbx,
                                           const double* gp, int64_t n) {
  const int m = p.k - 1;
  int nf = 0;
  for (int j = 0; j < m; ++j) nf += (cs[colmap[p.a_col + j]].flags & kCsNaN) ? 0 : 1;
  const int K = nf + 1;
  double G[kGramCols][kGramCols];
  for (int a = 0, e = 0; a < kGramCols; ++a)
    for (int bb = a; bb < kGramCols; ++bb, ++e) {
      double t = 0.0;
      if (bb < K)
        for (int x = 0; x < nbx; ++x) t += gp[(int64_t)x * kGramE + e];
      G[a][bb] = t;
      G[bb][a] = t;
    }
  double d0[kGramCols], g0[kGramCols], maxd = 0.0, floor = 1e-24;
  for (int a = 0; a < K; ++a) d0[a] = g0[a] = G[a][a];
  if (n > 0) {
    int f = 0;
    for (int j = 0; j < m; ++j) {
      const ColStat& st = cs[colmap[p.a_col + j]];
      if (!(st.flags & kCsNaN)) d0[f++] = st.sumsq;
    }
    d0[K - 1] = (double)n;
    floor *= (double)(K << 2 * (K - 1));
  }
  for (int a = 0; a < K; ++a) maxd = fmax(maxd, d0[a]);
  int piv[kGramCols];
  for (int a = 0; a < K; ++a) piv[a] = a;
  if (!(maxd > 0.0 && maxd < 1e300)) return 0;
  for (int s2 = 0; s2 < K; ++s2) {
    int q = s2;
    for (int j = s2 + 1; j < K; ++j)
      if (G[j][j] > G[q][q]) q = j;
    const double dp = G[q][q];
    if (!(dp > 1e-8 * d0[piv[q]]) || !(dp > floor * maxd)) return dp < 1e-13 * g0[piv[q]] ? -1 : 0;
    if (q != s2) {
      for (int j = 0; j < K; ++j) { const double t = G[s2][j]; G[s2][j] = G[q][j]; G[q][j] = t; }
      for (int j = 0; j < K; ++j) { const double t = G[j][s2]; G[j][s2] = G[j][q]; G[j][q] = t; }
      const int t = piv[s2]; piv[s2] = piv[q]; piv[q] = t;
    }
    const double l = sqrt(dp);
    for (int a = s2 + 1; a < K; ++a) G[a][s2] /= l;
    for (int a = s2 + 1; a < K; ++a)
      for (int bb = s2 + 1; bb <= a; ++bb) {
        G[a][bb] -= G[a][s2] * G[bb][s2];
        G[bb][a] = G[a][bb];
      }
  }
  return 1;
}

__device__ __forceinline__ void settle_candidate(const DevBatch& b, int c, PlainCand* pc, bool ok, double* coefs,
                                                 rrg_result* res, uint32_t* decided) {
  if (!ok) {
    pc[c].pad = 0;
    return;
  }
  const int k = pc[c].k;
  double* out = coefs + b.cands[c].coef_offset;
  for (int j = 0; j < k; ++j) out[j] = __longlong_as_double(0x7ff8000000000000ll);
  res[c].rank = k;
  pc[c].pad = 1;
  atomicAdd(decided, 1u);
}

__global__ void nan_gram_decide_kernel(DevBatch b, const int32_t* list, int cnt, PlainCand* pc, const int32_t* colmap,
                                       const ColStat* cs, int nbx, const double* gpart, double* coefs,
                                       rrg_result* res, uint32_t* decided, const int32_t* dcount) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= cnt || (dcount && i >= *dcount)) return;
  const int c = list[i];
  if (!(pc[c].pad & 2)) return;
  settle_candidate(b, c, pc, gram_certifies(pc[c], colmap, cs, nbx, gpart + (int64_t)i * nbx * kGramE, 0) > 0, coefs,
                   res, decided);
}

// The three above for one candidate a block: the certificate from kGramSample
// rows in eight runs spread over the dataset where the columns' norms are known
// (sums), else, or where that fails, from all rows if they are few (all_rows);
// what is still open keeps pad = 2.
constexpr int kGramSample = 2048;
__global__ void __launch_bounds__(256) nan_settle_kernel(DevBatch b, const int32_t* list, int cnt, PlainCand* pc,
                                                         const int32_t* colmap, const ColStat* cs, const double* T,
                                                         int64_t n, int64_t n_pad, double* coefs, rrg_result* res,
                                                         uint32_t* decided, const int32_t* dcount, bool sums,
                                                         bool all_rows) {
  __shared__ double red[8][kGramE], g[kGramE];
  __shared__ int pad;
  after_previous();
  if (dcount && (int)blockIdx.x >= *dcount) return;
  const int c = list[blockIdx.x];
  const PlainCand p = pc[c];
  if (threadIdx.x == 0) {
    pad = classify_candidate(b, c, p, colmap, cs, n, coefs, res, decided);
    if (pad) pc[c].pad = pad;
  }
  __syncthreads();
  if (pad != 2) return;
  if (sums && n > kGramSample) {
    gram_block(p, colmap, cs, T, n_pad, kGramSample / 256, [&](int64_t s) { return n * s / (kGramSample / 256); }, n,
               red, g);
    __syncthreads();
    if (threadIdx.x == 0) {
      const int r = gram_certifies(p, colmap, cs, 1, g, n);
      // dependent on the sample: most likely on all rows, and the QR's to find
      // (8192 random trees' re-scoring with its evaluation 13.9 ms, 14.8 with the
      // Gram matrix of all rows for these)
      if (r) settle_candidate(b, c, pc, r > 0, coefs, res, decided);
      pad = r ? 1 : 2;
    }
    __syncthreads();
    if (pad == 1) return;
  }
  if (!all_rows) return;
  gram_block(p, colmap, cs, T, n_pad, (n + 255) / 256, [](int64_t s) { return 256 * s; }, n, red, g);
  __syncthreads();
  if (threadIdx.x == 0) settle_candidate(b, c, pc, gram_certifies(p, colmap, cs, 1, g, 0) > 0, coefs, res, decided);
}

constexpr int64_t kGramRows = 32768;  // rows a block
static int nan_gram_blocks(int64_t n) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(16, (n + kGramRows - 1) / kGramRows));
}
size_t nan_gram_bytes(int64_t n, int cnt) {
  const int nbx = nan_gram_blocks(n);
  return nbx == 1 ? 1 : sizeof(double) * (size_t)cnt * nbx * kGramE;
}
bool launch_nan_settle(const DevBatch& b, const DevData& ds, const int32_t* list, int cnt, PlainCand* pc,
                       const int32_t* colmap, const ColStat* cs, bool sums, const double* T, double* gpart,
                       double* coefs, rrg_result* res, uint32_t* decided, const int32_t* dcount, cudaStream_t st,
                       int64_t* launches) {
  if (cnt <= 0) return true;
  // Up to kGramRows rows one launch settles every candidate.  Above, what the
  // sample leaves open goes over all rows with several blocks a candidate.
  // (A lone candidate of 150 rows is launches and latency.  The sample, against all
  // rows at once: 765 candidates at 20011 rows 0.06 against 0.28 ms; 2048 random
  // trees at 100k rows, with the evaluation, 6.9 against 7.4.)
  const int nbx = nan_gram_blocks(ds.n);
  *launches += 1;
  if (!launch_next(true, nan_settle_kernel, dim3(cnt), 256, 0, st, b, list, cnt, pc, colmap, cs, T, ds.n, ds.n_pad,
                   coefs, res, decided, dcount, sums, nbx == 1))
    return launch_ok("nan_settle");
  if (nbx == 1) return launch_ok("nan_settle");
  nan_gram_kernel<<<dim3(cnt, nbx), 256, 0, st>>>(list, cnt, pc, colmap, cs, T, ds.n, ds.n_pad, gpart, dcount);
  nan_gram_decide_kernel<<<(cnt + 127) / 128, 128, 0, st>>>(b, list, cnt, pc, colmap, cs, nbx, gpart, coefs, res,
                                                            decided, dcount);
  *launches += 2;
  return launch_ok("nan_gram");
}

size_t plain_eval_smem(int levels, int words) {
  return (size_t)levels * 256 * sizeof(double) + (size_t)words * sizeof(uint32_t);
}

}  // namespace rrd
