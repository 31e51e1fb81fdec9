// Column-pivoted QR least squares of the plain FP64 path over whole-GPU
// passes: the factorisation of ColPivHouseholderQR::computeInPlace
// (eigen/Eigen/src/QR/ColPivHouseholderQR.h:482-575) and its least-squares
// solve (:577-608), with makeHouseholder / applyHouseholderOnTheLeft semantics
// (eigen/Eigen/src/Householder/Householder.h:67-133), every sum in the QSUM
// order of csrc/common/rr_sum.h.
//
// A candidate's rows are cut into chunks of RR_CHUNK rows.  A pass is one
// launch over (candidate, chunk, column group) items; an item is a 256-thread
// block whose thread t is QSUM lane t of the chunk (its rows i with
// i mod 256 = t, in increasing order), so the block folds its lanes into the
// chunk's totals.  The last block of a candidate to finish a pass (a ticket
// counter) adds the chunk totals in chunk order and does the scalar work of the
// step (pivot choice, rank rule, Householder scalars, norm down-dating):
//
//   sums   once per table column, whatever the number of candidates that read
//          it: its sum of squares over rows >= 0 and over rows >= 1, kept with
//          the column's statistics
//   begin  one warp per candidate: norms from those sums, step 0's pivot and
//          reflector
//   A(kk)  the dots v . a_j of the Householder vector v (the pivot's tail over
//          c0 - beta) with the remaining columns; last block: row kk of R,
//          -tmp_j, down-dating, and the pivot of step kk + 1 when no norm must
//          be recomputed
//   B(kk)  a_j += (tau v_i) (-tmp_j), and the sums of squares of updated
//          columns that step kk + 1 needs (recomputed norms over rows >= kk + 1,
//          pivot tails over rows >= kk + 2); last block: step kk + 1's pivot
//          and reflector
//   solve  back substitution with R and the transformed y
//
// What is not done: step 0 reads the table's columns, y and the column of ones
// where they are (B(0) writes the working columns, so nothing is copied first);
// v is not stored (both passes form it from the pivot's column, a quotient by
// one divisor on the integer pipes, csrc/common/fp64_int.h); the last step
// updates nothing (row kk of y is all the solve reads); and a rank cut ends the
// factorisation, since later steps change neither the rank nor the leading
// block that the solve reads.
//
// A sum over rows >= kk + 2 differs from the one over rows >= kk + 1 only in
// the lane that owns row kk + 1, whose chain starts there: that lane forms
// the shorter chain too, and the chunk holding row kk + 1 is folded twice.
//
// Bound: the FP64 pipe (one warp instruction holds it 17 to 20 cycles).  A
// four-column candidate (three factors and the free term) takes 25 FP64
// instructions a row (dots 10, updates 9, tails 3, its share of the column
// sums) against 47 with the copy, a stored v and native quotients, and moves
// about 32 columns against 51.  Measured on GB300 (QR phase, before / now): a
// 660-candidate round at 1M rows, mostly three columns, 52.5 / 18.7 ms (13.3 ms
// at 17 cycles for its 13 FP64 instructions a row); the re-scored candidates
// of eight certified rounds at 1M rows 51.0 / 28.9 ms; 765 candidates at 20011
// rows 4.02 / 2.47 ms; one candidate at 1M rows 0.59 / 0.29 ms.
// Rows held per lane 8 (A) and 4 (B) at four resident blocks: 19.4 ms; 8 and 8
// 19.8, 4 and 4 19.9, three resident blocks 21.6.
#include <cfloat>
#include <cstdint>

#include "../common/error.h"
#include "../common/fp64_int.h"
#include "../common/rr_sum.h"
#include "common.cuh"
#include "plain.cuh"
#include "qr_chunk.cuh"
#include "qr_ops.cuh"
#include "reduce.cuh"

namespace rrd {

namespace {

constexpr int kQC = RR_CHUNK;
constexpr double kDowndateThr = 1.4901161193847656e-08;  // sqrt(DBL_EPSILON)
// rows of a lane handled together (loads in flight per column) in pass A and
// the column sums, and in pass B
constexpr int kRowsA = 8;
constexpr int kRowsB = 4;
// chunk totals staged together by a candidate's last block
constexpr int kStage = 2048;

__device__ __forceinline__ int job_count(const QrJob& j) {
  if (!j.dcount) return j.n_list;
  const int n = *j.dcount - j.list_off;
  return n < 0 ? 0 : (n > j.n_list ? j.n_list : n);
}

__device__ __forceinline__ double* wcol(const QrJob& j, int t, int c, int s) {
  const int64_t base = j.slot_cols > 0 ? (int64_t)t * j.slot_cols : j.pc[c].m_col;
  return j.M + (base + s) * j.ds.n_pad;
}

// Storage column s of the design [factors | 1 | y] as step 0 finds it; NULL:
// the column of ones.
__device__ __forceinline__ const double* design_col(const QrJob& j, int c, int k, int s) {
  if (s == k) return j.ds.y64;
  return s == k - 1 ? nullptr : factor_column(j.A, j.ds.n_pad, j.pc[c].a_col, s, j.colmap);
}

// chunk total of sum slot s; row nch holds the shorter-range variant
__device__ __forceinline__ double* part_at(const QrJob& j, int t, int row, int s) {
  return j.part + ((int64_t)t * (j.nch + 1) + row) * j.max_cols + s;
}
// R of candidate t: row kk, storage column s
__device__ __forceinline__ double* r_at(const QrJob& j, int t, int kk, int s) {
  return j.rmat + ((int64_t)t * j.max_cols + kk) * j.max_cols + s;
}

// Totals of sum slots [0, cnt) in chunk order from 0 into out (shared) and,
// when sp >= 0, the totals with chunk sp's variant in its place into out_sp.
// The totals are staged in buf (kStage shared doubles) by the whole block, and
// a thread adds one of them up: an FP64 addition that waits for the one before
// takes about 95 cycles, so the ordered sums run side by side.
__device__ __forceinline__ void chunk_totals(const QrJob& j, int t, int cnt, int sp, double* buf, double* out,
                                             double* out_sp) {
  const int nch = j.nch;
  const int per = nch + 1 <= kStage ? kStage / (nch + 1) : 0;  // slots staged at once
  const int sums = sp >= 0 ? 2 : 1;
  for (int s0 = 0; s0 < cnt; s0 += per > 0 ? per : cnt) {
    const int ns = per > 0 && per < cnt - s0 ? per : cnt - s0;
    if (per > 0) {
      for (int i = threadIdx.x; i < ns * (nch + 1); i += blockDim.x) {
        const int row = i % (nch + 1);
        if (row < nch || sp >= 0) buf[i] = __ldcg(part_at(j, t, row, s0 + i / (nch + 1)));
      }
      __syncthreads();
    }
    for (int x = threadIdx.x; x < ns * sums; x += blockDim.x) {
      const int s = x / sums, skip = x % sums ? sp : -1;
      double tot = 0.0;
      for (int ch = 0; ch < nch; ++ch) {
        const int row = ch == skip ? nch : ch;
        tot = __dadd_rn(tot, per > 0 ? buf[s * (nch + 1) + row] : __ldcg(part_at(j, t, row, s0 + s)));
      }
      (x % sums ? out_sp : out)[s0 + s] = tot;
    }
    __syncthreads();
  }
}

// After an item's chunk totals are written: true in the block that finishes
// the candidate's pass last (every other block's writes are then visible)
__device__ __forceinline__ bool last_block(unsigned int* ticket, int items, int* s_flag) {
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) *s_flag = atomicAdd(ticket, 1u) == (unsigned)(items - 1) ? 1 : 0;
  __syncthreads();
  const bool last = *s_flag != 0;
  if (last) __threadfence();
  return last;
}

// Businger-Golub pivot of step kk (largest down-dated norm, first index on
// ties), the rank rule of ColPivHouseholderQR.h:504-511, and the swap; a cut
// ends the factorisation (size = rank)
__device__ void select_pivot(QrState* S, int kk, double rows) {
  int big = kk;
  double bign = S->nupd[kk];
  for (int j = kk + 1; j < S->k; ++j)
    if (fi_lt(bign, S->nupd[j])) {
      bign = S->nupd[j];
      big = j;
    }
  if (fi_lt(fi_mul(bign, bign), fi_mul(S->thr_helper, rows - kk))) {
    S->size = kk;
    return;
  }
  if (big != kk) {
    double t = S->nupd[kk]; S->nupd[kk] = S->nupd[big]; S->nupd[big] = t;
    t = S->ndir[kk]; S->ndir[kk] = S->ndir[big]; S->ndir[big] = t;
    int p = S->pos2col[kk]; S->pos2col[kk] = S->pos2col[big]; S->pos2col[big] = p;
  }
}

// makeHouseholder of the pivot from its diagonal entry and tail sum of squares
__device__ void householder_scalars(QrState* S, double c0, double tail_sq) {
  if (tail_sq <= DBL_MIN) {
    S->tau = 0.0;
    S->beta = c0;
    S->den = 1.0;
    S->tau_zero = 1;
  } else {
    double beta = fi_sqrt(__dadd_rn(fi_mul(c0, c0), tail_sq));
    if (c0 >= 0.0) beta = -beta;
    const double den = __dsub_rn(c0, beta);
    S->den = den;
    S->tau = fi_div(-den, beta);
    S->beta = beta;
    S->tau_zero = 0;
  }
}

// Columns of one item.  Four: the accumulators, a column's rows and the
// pivot's fit 64 registers (four resident blocks); a wider candidate takes
// several items a chunk, each forming v again.
constexpr int CG = 4;
constexpr int kMinBlocks = 4;

// Columns an item takes: CG, or fewer while the pass has less than two items
// per block of the grid (a lone candidate at 1M rows has 62 chunks; one column
// an item then spreads it over four times the blocks)
__device__ __forceinline__ int cols_per_item(int64_t chunks, int width) {
  int c = CG;
  while (c > 1 && chunks * ((width + c - 1) / c) < 2 * (int64_t)gridDim.x) c >>= 1;
  return c;
}

// Calls body(s0, full) for the lane's rows [lo, hi) of the chunk at r0 in
// sub-chunks of U rows a lane, in order; `full`: every row of it is in range.
template <int U, class F>
__device__ __forceinline__ void sub_chunks(int64_t r0, int64_t lo, int64_t hi, F&& body) {
  for (int64_t s0 = r0; s0 < r0 + kQC && s0 < hi; s0 += 256 * U) {
    if (s0 + 256 * U <= lo) continue;
    body(s0, s0 >= lo && s0 + 256 * U <= hi);
  }
}

// U rows of a column (ones when col is NULL); rows out of [lo, hi) read 0
template <int U>
__device__ __forceinline__ void load_rows(const double* col, int64_t i0, int64_t lo, int64_t hi, bool full,
                                          double (&v)[U]) {
  if (!col) {
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = 1.0;
  } else if (full) {
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = __ldcg(col + i0 + 256 * u);
  } else {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = i0 + 256 * u;
      v[u] = i >= lo && i < hi ? __ldcg(col + i) : 0.0;
    }
  }
}

}  // namespace

// ------------------------------------------------------------- column sums --
// A column's totals from its chunk totals pt[0 .. nch] (the last one chunk 0's
// without row 0), by its last block.
__device__ __forceinline__ void col_sums_finish(const double* pt, int nch, double* buf, ColStat* cs) {
  for (int i = threadIdx.x; i <= nch && i < kStage; i += blockDim.x) buf[i] = __ldcg(pt + i);
  __syncthreads();
  if (threadIdx.x == 0 || threadIdx.x == 32) {
    double tot = 0.0;
    for (int i = 0; i < nch; ++i) {
      const int x = threadIdx.x == 32 && i == 0 ? nch : i;
      tot = __dadd_rn(tot, x < kStage ? buf[x] : __ldcg(pt + x));
    }
    if (threadIdx.x == 0) cs->sumsq = tot;
    else cs->tailsq = tot;
  }
  if (threadIdx.x == 0) cs->ticket = 0;
  __syncthreads();
}

__global__ void __launch_bounds__(256) col_sums_kernel(const double* T, int64_t n, int64_t n_pad, const int32_t* cols,
                                                       int n_cols, const int32_t* dcount, ColStat* cst, double* part) {
  __shared__ double red[8], outA[1], outB[1], buf[kStage];
  __shared__ int s_flag;
  const int cnt = dcount ? min(*dcount, n_cols) : n_cols;
  const int nch = (int)((n + kQC - 1) / kQC);
  const int64_t items = (int64_t)cnt * nch;
  for (int64_t it = blockIdx.x; it < items; it += gridDim.x) {
    const int t = (int)(it / nch), ch = (int)(it % nch);
    const int32_t c = cols[t];
    if (cst[c].flags & kCsStop) {  // a NaN beyond row 0: not read
      if (ch == 0 && threadIdx.x == 0) cst[c].sumsq = cst[c].tailsq = __longlong_as_double(0x7ff8000000000000ll);
      continue;
    }
    const double* col = T + (int64_t)c * n_pad;
    const int64_t r0 = (int64_t)ch * kQC, hi = r0 + kQC < n ? r0 + kQC : n;
    const bool row0 = ch == 0 && threadIdx.x == 0;  // the lane owning row 0: also its chain without that row
    double p = 0.0, q = 0.0;
    sub_chunks<kRowsA>(r0, r0, hi, [&](int64_t s0, bool full) {
      double v[kRowsA];
      const int64_t i0 = s0 + threadIdx.x;
      load_rows(col, i0, r0, hi, full, v);
#pragma unroll
      for (int u = 0; u < kRowsA; ++u)
        if (full || i0 + 256 * u < hi) {
          p = __fma_rn(v[u], v[u], p);
          if (row0 && (u > 0 || s0 > 0)) q = __fma_rn(v[u], v[u], q);
        }
    });
    double* pt = part + (int64_t)t * (nch + 1);
    double va[1] = {p};
    fold_lanes<1>(va, 1, red, outA);
    if (ch == 0) {
      va[0] = row0 ? q : p;
      fold_lanes<1>(va, 1, red, outB);
    }
    if (threadIdx.x == 0) {
      pt[ch] = outA[0];
      if (ch == 0) pt[nch] = outB[0];
    }
    if (last_block(&cst[c].ticket, nch, &s_flag)) col_sums_finish(pt, nch, buf, cst + c);
  }
}

namespace {

// ------------------------------------------------------------------ begin --
// One warp per candidate: norms, thresholds, step 0's pivot and reflector.
__global__ void __launch_bounds__(128) qr_begin_kernel(QrJob j) {
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= job_count(j)) return;
  QrState* S = j.state + t;
  const int c = j.list[j.list_off + t];
  const rrg_cand cd = j.b.cands[c];
  const int k = j.pc[c].k;
  bool active = cd.mode == RRG_TUNED && !(j.pc[c].pad & 1) && k >= 1;
  if (active && k + 1 > j.max_cols) {
    if (lane == 0) atomicOr(j.status, ST_TOO_LARGE);
    active = false;
  }
  if (!active) {
    if (lane == 0) S->active = 0;
    return;
  }
  const double rows_d = (double)j.ds.n;
  for (int s = lane; s <= k; s += 32) {
    S->pos2col[s] = s;
    if (s < k) {
      const double sq = s == k - 1 ? rows_d : j.cst[j.colmap[j.pc[c].a_col + s]].sumsq;
      const double nr = __dsqrt_rn(sq);
      S->ndir[s] = nr;
      S->nupd[s] = nr;
    }
  }
  __syncwarp();
  if (lane != 0) return;
  S->active = 1;
  S->k = k;
  S->size = (int)(j.ds.n < k ? j.ds.n : k);
  S->ticket = 0;
  S->rec_any = 0;
  S->nsum = 0;
  double maxn = S->nupd[0];
  for (int s = 1; s < k; ++s)
    if (S->nupd[s] > maxn) maxn = S->nupd[s];
  S->thr_helper = __ddiv_rn(__dmul_rn(__dmul_rn(maxn, DBL_EPSILON), __dmul_rn(maxn, DBL_EPSILON)), rows_d);
  select_pivot(S, 0, rows_d);
  if (S->size == 0) return;
  const int ps = S->pos2col[0];
  const double* col = design_col(j, c, k, ps);
  const double tail = !col ? rows_d - 1.0 : j.cst[j.colmap[j.pc[c].a_col + ps]].tailsq;
  householder_scalars(S, col ? col[0] : 1.0, j.ds.n == 1 ? 0.0 : tail);
}

// Shared per-item view: the columns of the item's group.
struct ItemView {
  const double* src[CG];  // NULL: ones
  double* dst[CG];
  double ntmp[CG];
  int slot[CG];           // sum slot, or -1
};

// The whole state of a candidate between global and shared memory.
__device__ __forceinline__ void copy_state(QrState* dst, const QrState* src) {
  static_assert(sizeof(QrState) % 8 == 0, "copied by words");
  const unsigned long long* s = reinterpret_cast<const unsigned long long*>(src);
  unsigned long long* d = reinterpret_cast<unsigned long long*>(dst);
  for (int i = threadIdx.x; i < (int)(sizeof(QrState) / 8); i += blockDim.x) d[i] = s[i];
  __syncthreads();
}

// Shared memory of a candidate's last block.
struct Finish {
  QrState Ss;
  double buf[kStage], tot[kQrMaxCols], tail[kQrMaxCols];
  int8_t rec[kQrMaxCols];
};

// Pass A's scalar work, by a candidate's last block.
__device__ void passA_finish(Finish& F, const QrJob& j, int t, int c, int kk, bool upd) {
  // ---- last block: row kk (Householder.h:121-126), then down-dating
  QrState* S = j.state + t;
  copy_state(&F.Ss, S);
  const int k = F.Ss.k, nw = k - kk, ps = F.Ss.pos2col[kk];
  const int64_t rows = j.ds.n;
  if (upd) chunk_totals(j, t, nw, -1, F.buf, F.tot, nullptr);
  const int next = kk + 1;
  for (int q = threadIdx.x; q < nw; q += blockDim.x) {
    const int p = next + q, s = p < k ? F.Ss.pos2col[p] : k;
    const double* col = kk == 0 ? design_col(j, c, k, s) : wcol(j, t, c, s);
    const double qk = col ? __ldcg(col + kk) : 1.0;
    double a = qk;
    if (upd) {
      const double tmp = __dadd_rn(F.tot[q], qk);
      a = __dsub_rn(qk, fi_mul(F.Ss.tau, tmp));
      F.Ss.ntmp[s] = -tmp;
    } else if (rows - kk == 1) {
      a = __dmul_rn(qk, __dsub_rn(1.0, F.Ss.tau));  // a one-row tail
    }
    *r_at(j, t, kk, s) = a;
    // LAWN 176 norm down-dating (ColPivHouseholderQR.h:549-572); the
    // recomputations happen in pass B, which sums the updated columns
    int flag = 0;
    if (p < k && F.Ss.nupd[p] != 0.0) {
      const double nu = F.Ss.nupd[p];
      double temp = fi_div(fabs(a), nu);
      temp = fi_mul(__dadd_rn(1.0, temp), __dsub_rn(1.0, temp));
      temp = temp < 0.0 ? 0.0 : temp;
      const double ratio = fi_div(nu, F.Ss.ndir[p]);
      const double temp2 = fi_mul(temp, fi_mul(ratio, ratio));
      if (temp2 <= kDowndateThr) flag = 1;
      else F.Ss.nupd[p] = fi_mul(nu, fi_sqrt(temp));
    }
    F.rec[q] = (int8_t)flag;
    F.Ss.slot_of[s] = -1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    *r_at(j, t, kk, ps) = F.Ss.beta;
    int rec_any = 0, nsum = 0;
    for (int q = 0; q < nw - 1; ++q) rec_any |= F.rec[q];
    if (next < F.Ss.size) {
      if (rec_any) {
        // the pivot of step kk + 1 depends on the recomputed norms (and on
        // NaN norms through the scan's running maximum): the sums of every
        // remaining column, which a recomputation step can afford
        for (int p = next; p < k; ++p) {
          F.Ss.slot_of[F.Ss.pos2col[p]] = nsum;
          F.Ss.sum_norm[nsum++] = F.rec[p - next];
        }
      } else {
        select_pivot(&F.Ss, next, (double)rows);
        if (next < F.Ss.size) {
          F.Ss.slot_of[F.Ss.pos2col[next]] = 0;
          F.Ss.sum_norm[0] = 0;
          nsum = 1;
        }
      }
    }
    F.Ss.rec_any = rec_any;
    F.Ss.nsum = nsum;
    F.Ss.ticket = 0;
  }
  __syncthreads();
  copy_state(S, &F.Ss);
}

// Pass B's.
__device__ void passB_finish(Finish& F, const QrJob& j, int t, int c, int kk) {
  // ---- the candidate's last block: totals, then step kk + 1's scalars
  QrState* S = j.state + t;
  copy_state(&F.Ss, S);
  const int k = F.Ss.k, next = kk + 1;
  const int64_t rows = j.ds.n;
  const int nsum = F.Ss.nsum;
  chunk_totals(j, t, nsum, next / kQC, F.buf, F.tot, F.tail);
  if (threadIdx.x == 0) {
    if (F.Ss.rec_any) {
      // recomputed norms (ColPivHouseholderQR.h:566-569)
      for (int p = next; p < k; ++p) {
        const int q = F.Ss.slot_of[F.Ss.pos2col[p]];
        if (q >= 0 && F.Ss.sum_norm[q]) {
          F.Ss.ndir[p] = fi_sqrt(F.tot[q]);
          F.Ss.nupd[p] = F.Ss.ndir[p];
        }
      }
      select_pivot(&F.Ss, next, (double)rows);
    }
    if (next < F.Ss.size) {
      const int np = F.Ss.pos2col[next], q = F.Ss.slot_of[np];
      if (q < 0) {
        atomicOr(j.status, ST_QR_STATE);
        F.Ss.active = 0;
      } else {
        householder_scalars(&F.Ss, __ldcg(wcol(j, t, c, np) + next), rows - next == 1 ? 0.0 : F.tail[q]);
      }
    }
    F.Ss.ticket = 0;
  }
  __syncthreads();
  copy_state(S, &F.Ss);
}

// ------------------------------------------------------------------ A(kk) --
__global__ void __launch_bounds__(256, kMinBlocks) qr_passA_kernel(QrJob j, int kk, int width) {
  __shared__ ItemView V;
  __shared__ double red[8 * CG], outA[CG];
  __shared__ int s_flag;
  __shared__ Finish F;
  const int cnt = job_count(j);
  const int64_t rows = j.ds.n;
  const int cpi = cols_per_item((int64_t)cnt * j.nch, width);
  const int gmax = (width + cpi - 1) / cpi;
  const int64_t items = (int64_t)cnt * j.nch * gmax;
  for (int64_t it = blockIdx.x; it < items; it += gridDim.x) {
    const int g = (int)(it % gmax), ch = (int)(it / gmax % j.nch), t = (int)(it / ((int64_t)gmax * j.nch));
    QrState* S = j.state + t;
    if (!S->active || kk >= S->size) continue;  // uniform over the block
    const int k = S->k, nw = k - kk, groups = (nw + cpi - 1) / cpi;
    if (g >= groups) continue;
    const int c = j.list[j.list_off + t];
    const int q0 = g * cpi, gc = min(cpi, nw - q0);
    const bool upd = !S->tau_zero && rows - kk > 1;
    const int ps = S->pos2col[kk];
    const double* piv = kk == 0 ? design_col(j, c, k, ps) : wcol(j, t, c, ps);
    const fi_divisor den = fi_divisor_of(S->den);
    if (threadIdx.x < gc) {
      const int p = kk + 1 + q0 + threadIdx.x, s = p < k ? S->pos2col[p] : k;
      V.src[threadIdx.x] = kk == 0 ? design_col(j, c, k, s) : wcol(j, t, c, s);
    }
    __syncthreads();
    if (upd) {
      const int64_t r0 = (int64_t)ch * kQC;
      const int64_t lo = r0 > kk + 1 ? r0 : kk + 1, hi = r0 + kQC < rows ? r0 + kQC : rows;
      double pa[CG];
#pragma unroll
      for (int q = 0; q < CG; ++q) pa[q] = 0.0;
      sub_chunks<kRowsA>(r0, lo, hi, [&](int64_t s0, bool full) {
        const int64_t i0 = s0 + threadIdx.x;
        double v[kRowsA], a[kRowsA];
        load_rows(piv, i0, lo, hi, full, v);
        load_rows(V.src[0], i0, lo, hi, full, a);
        // the Householder vector (Householder.h:83-90): the tail over c0 - beta
#pragma unroll
        for (int u = 0; u < kRowsA; ++u) v[u] = fi_div_by(v[u], &den);
#pragma unroll
        for (int q = 0; q < CG; ++q) {
          if (q >= gc) break;
          if (q > 0) load_rows(V.src[q], i0, lo, hi, full, a);
          double acc = pa[q];
          if (full) {
#pragma unroll
            for (int u = 0; u < kRowsA; ++u) acc = __fma_rn(v[u], a[u], acc);
          } else {
#pragma unroll
            for (int u = 0; u < kRowsA; ++u) {
              const int64_t i = i0 + 256 * u;
              if (i >= lo && i < hi) acc = __fma_rn(v[u], a[u], acc);
            }
          }
          pa[q] = acc;
        }
      });
      fold_lanes<CG>(pa, gc, red, outA);
      if (threadIdx.x < gc) *part_at(j, t, ch, q0 + threadIdx.x) = outA[threadIdx.x];
    }
    if (!last_block(&S->ticket, j.nch * groups, &s_flag)) continue;
    passA_finish(F, j, t, c, kk, upd);
  }
}

// ------------------------------------------------------------------ B(kk) --
__global__ void __launch_bounds__(256, kMinBlocks) qr_passB_kernel(QrJob j, int kk, int width) {
  __shared__ ItemView V;
  __shared__ double red[8], outA[1], outB[1];
  __shared__ int s_flag;
  __shared__ Finish F;
  const int cnt = job_count(j);
  const int64_t rows = j.ds.n;
  const int next = kk + 1;
  const int cpi = cols_per_item((int64_t)cnt * j.nch, width);
  const int gmax = (width + cpi - 1) / cpi;
  const int64_t items = (int64_t)cnt * j.nch * gmax;
  for (int64_t w = blockIdx.x; w < items; w += gridDim.x) {
    const int64_t it = items - 1 - w;  // pass A's last items first: what they read is still in L2
    const int g = (int)(it % gmax), ch = (int)(it / gmax % j.nch), t = (int)(it / ((int64_t)gmax * j.nch));
    QrState* S = j.state + t;
    if (!S->active || next >= S->size) continue;  // the last step updates nothing that is read
    const int k = S->k, nw = k - kk, groups = (nw + cpi - 1) / cpi;
    if (g >= groups) continue;
    const int c = j.list[j.list_off + t];
    const int q0 = g * cpi, gc = min(cpi, nw - q0);
    const bool upd = !S->tau_zero && rows - kk > 1;
    const int ps = S->pos2col[kk];
    const double* piv = kk == 0 ? design_col(j, c, k, ps) : wcol(j, t, c, ps);
    const fi_scaled tq = fi_scaled_of(S->tau, S->den);
    if (threadIdx.x < gc) {
      const int p = next + q0 + threadIdx.x, s = p < k ? S->pos2col[p] : k;
      V.dst[threadIdx.x] = wcol(j, t, c, s);
      V.src[threadIdx.x] = kk == 0 ? design_col(j, c, k, s) : V.dst[threadIdx.x];
      V.ntmp[threadIdx.x] = S->ntmp[s];
      V.slot[threadIdx.x] = S->slot_of[s];
    }
    __syncthreads();
    const int64_t r0 = (int64_t)ch * kQC;
    const int64_t lo = r0 > next ? r0 : next, hi = r0 + kQC < rows ? r0 + kQC : rows;
    const bool write = upd || kk == 0;
    double ps2[CG];
#pragma unroll
    for (int q = 0; q < CG; ++q) ps2[q] = 0.0;
    sub_chunks<kRowsB>(r0, lo, hi, [&](int64_t s0, bool full) {
      const int64_t i0 = s0 + threadIdx.x;
      double tv[kRowsB], a[kRowsB];
      if (upd) load_rows(piv, i0, lo, hi, full, tv);
      load_rows(V.src[0], i0, lo, hi, full, a);
      if (upd) {
#pragma unroll
        for (int u = 0; u < kRowsB; ++u) tv[u] = fi_scaled_quot(tv[u], &tq);  // tau v_i
      }
#pragma unroll
      for (int q = 0; q < CG; ++q) {
        if (q >= gc) break;
        double* dst = V.dst[q];
        const double nt = V.ntmp[q];
        const bool sum = V.slot[q] >= 0;
        if (q > 0) load_rows(V.src[q], i0, lo, hi, full, a);
        if (upd) {
#pragma unroll
          for (int u = 0; u < kRowsB; ++u) a[u] = __fma_rn(tv[u], nt, a[u]);
        }
        double acc = ps2[q];
        if (full) {
          if (write) {
#pragma unroll
            for (int u = 0; u < kRowsB; ++u) dst[i0 + 256 * u] = a[u];
          }
          if (sum) {
#pragma unroll
            for (int u = 0; u < kRowsB; ++u) acc = __fma_rn(a[u], a[u], acc);
          }
        } else {
#pragma unroll
          for (int u = 0; u < kRowsB; ++u) {
            const int64_t i = i0 + 256 * u;
            if (i >= lo && i < hi) {
              if (write) dst[i] = a[u];
              if (sum) acc = __fma_rn(a[u], a[u], acc);
            }
          }
        }
        ps2[q] = acc;
      }
    });
    // the sums' chunk totals; in the chunk holding row kk + 1 also without
    // that row (the lane owning it forms its chain again)
    const bool sp_chunk = next >= r0 && next < r0 + kQC;
    const bool sp_lane = sp_chunk && (next & 255) == (int)threadIdx.x;
#pragma unroll
    for (int q = 0; q < CG; ++q) {
      if (q >= gc) break;
      const int sl = V.slot[q];
      if (sl < 0) continue;  // uniform
      double va[1] = {ps2[q]};
      fold_lanes<1>(va, 1, red, outA);
      if (sp_chunk) {
        if (sp_lane) {
          va[0] = 0.0;
          const double* col = write ? V.dst[q] : V.src[q];
          for (int64_t i = next + 256; i < hi; i += 256) {
            const double x = __ldcg(col + i);
            va[0] = __fma_rn(x, x, va[0]);
          }
        }
        fold_lanes<1>(va, 1, red, outB);
      }
      if (threadIdx.x == 0) {
        *part_at(j, t, ch, sl) = outA[0];
        if (sp_chunk) *part_at(j, t, j.nch, sl) = outB[0];
      }
    }
    if (!last_block(&S->ticket, j.nch * groups, &s_flag)) continue;
    passB_finish(F, j, t, c, kk);
  }
}

// ------------------------------------------------------------------ solve --
__global__ void qr_solve_kernel(QrJob j) {
  const int cnt = job_count(j);
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < cnt; t += gridDim.x * blockDim.x) {
    const QrState* S = j.state + t;
    if (!S->active) continue;
    const int c = j.list[j.list_off + t];
    const rrg_cand cd = j.b.cands[c];
    const int k = S->k, r = S->size;
    double cvec[kQrMaxCols];
    for (int i = 0; i < r; ++i) cvec[i] = *r_at(j, t, i, k);
    for (int kk = r - 1; kk >= 0; --kk) {
      const int s = S->pos2col[kk];
      cvec[kk] = __ddiv_rn(cvec[kk], *r_at(j, t, kk, s));
      for (int i = 0; i < kk; ++i) cvec[i] = __dsub_rn(cvec[i], __dmul_rn(cvec[kk], *r_at(j, t, i, s)));
    }
    double* out = j.coefs + cd.coef_offset;
    for (int q = 0; q < k; ++q) out[q] = 0.0;
    for (int i = 0; i < r; ++i) out[S->pos2col[i]] = cvec[i];
    j.res[c].rank = r;
    if (j.count_bytes) {
      // every remaining column read and written once per step, the pivot's
      // and y read in the last
      double cols = r > 0 ? 2.0 : 0.0;
      for (int kk = 0; kk + 1 < r; ++kk) cols += 2.0 * (double)(k + 1 - kk);
      atomicAdd(reinterpret_cast<unsigned long long*>(j.status + kStatusQrBytes),
                (unsigned long long)(cols * 8.0 * (double)j.ds.n));
    }
  }
}

}  // namespace

size_t qr_chunk_scratch_bytes(int64_t n_list, int64_t rows, int max_cols) {
  const int64_t nch = (rows + kQC - 1) / kQC;
  const size_t st = round_up(sizeof(QrState) * (size_t)n_list, 256);
  return st + sizeof(double) * (size_t)n_list * (size_t)max_cols * (size_t)(nch + 1 + max_cols);
}

void qr_chunk_bind(QrJob& job, void* scratch) {
  job.nch = (int)((job.ds.n + kQC - 1) / kQC);
  const size_t st = round_up(sizeof(QrState) * (size_t)job.n_list, 256);
  job.state = static_cast<QrState*>(scratch);
  job.part = reinterpret_cast<double*>(static_cast<char*>(scratch) + st);
  job.rmat = job.part + (size_t)job.n_list * (size_t)(job.nch + 1) * (size_t)job.max_cols;
}

int qr_chunk_blocks_per_sm() {
  int a = 0, b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, qr_passA_kernel, 256, 0) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, qr_passB_kernel, 256, 0) != cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  const int m = a < b ? a : b;
  return m < 1 ? 1 : m;
}

bool launch_col_sums(const double* T, const DevData& ds, const int32_t* cols, int n_cols, const int32_t* dcount,
                     ColStat* cst, double* part, int max_blocks, cudaStream_t st) {
  if (n_cols <= 0) return true;
  const int64_t items = (int64_t)n_cols * ((ds.n + kQC - 1) / kQC);
  const int grid = (int)(items < max_blocks ? items : max_blocks);
  col_sums_kernel<<<grid < 1 ? 1 : grid, 256, 0, st>>>(T, ds.n, ds.n_pad, cols, n_cols, dcount, cst, part);
  return launch_ok("column sums");
}

bool launch_qr_chunked(const QrJob& job, int max_blocks, cudaStream_t st, int64_t* launches) {
  if (job.n_list <= 0) return true;
  if (job.max_cols > kQrMaxCols || job.max_cols < 2) {
    rrc::set_error("QR launch: column bound outside the kernel's range");
    return false;
  }
  const int steps = job.max_steps > 0 && job.max_steps < job.max_cols ? job.max_steps : job.max_cols - 1;
  qr_begin_kernel<<<(job.n_list + 3) / 4, 128, 0, st>>>(job);
  if (!launch_ok("QR begin")) return false;
  for (int kk = 0; kk < steps; ++kk) {
    // a candidate of k columns reaches k - kk of them (the free term and y
    // included); at most steps - kk over the job
    const int width = steps - kk;
    const int64_t items = (int64_t)job.n_list * job.nch * width;
    const int blocks = (int)(items < max_blocks ? items : max_blocks);
    qr_passA_kernel<<<blocks < 1 ? 1 : blocks, 256, 0, st>>>(job, kk, width);
    if (kk + 1 < steps) qr_passB_kernel<<<blocks < 1 ? 1 : blocks, 256, 0, st>>>(job, kk, width);
    if (!launch_ok("QR step passes")) return false;
  }
  const int sb = (int)((job.n_list + 127) / 128);
  qr_solve_kernel<<<sb < 1 ? 1 : sb, 128, 0, st>>>(job);
  if (!launch_ok("QR solve")) return false;
  if (launches) *launches += 1 + 2 * (int64_t)steps;
  return true;
}

}  // namespace rrd
