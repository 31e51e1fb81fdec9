// Kernels of the plain FP64 path (plain.cu).
#pragma once
#include "common.cuh"

namespace rrd {

constexpr int kMaxCodeSmem = 4096;  // words of a block's program staging; the last one flags a NaN

// A table column of n rows is evaluated in at least this many pieces, so that a
// level ends evenly (columns differ in cost by two orders of magnitude) and the
// pieces after one with a NaN find it.  4096 rows a piece: 2048 random trees at
// 100k rows 26.4 ms with one piece a column, 16.8 with 16384 rows a piece, 15.4
// with 4096, 14.7 with 2048; 627 columns of 1M rows 16.9, 14.5, 14.7, 15.1.
constexpr int64_t kEvalRows = 4096;
inline int64_t eval_pieces(int64_t n) { return n <= kEvalRows ? 1 : (n + kEvalRows - 1) / kEvalRows; }

// Rows to evaluate; live (may be NULL): [column] 0 where nothing counts any more.
struct EvalRows {
  int64_t lo, hi;
  const uint8_t* live;
  // the launch's shared memory: spill levels, words of program staging
  int32_t levels = RRG_MAX_STACK, words = kMaxCodeSmem;
};
// Shared columns, most of a batch of unlike trees, count only as long as a
// factor that reads them does.  So where there are many, the first kFirstRows
// rows of all levels are evaluated first, live_columns_kernel finds what still
// counts, and the other rows of the other columns are left out.  (They are
// nobody's: a shared column lives for one round.)  2048 random trees at 100k rows,
// 2100 shared columns: FP64 evaluation 7.4 ms, in one part 14.3 (8.0 with 4096
// first rows, 8.4 with 8192); 8192 trees: double-float 6.5, in one part 13.6.
// Where few columns are shared, or the work is below about 2 ms, the second pass
// over the levels could cost more than it saves.
constexpr int64_t kFirstRows = 1024;
inline bool eval_two_parts(int64_t n, int64_t shared, int64_t columns) {
  return n >= 16 * kFirstRows && shared * 4 >= columns && shared * n >= (int64_t(1) << 26);
}
struct ColStat;
struct LiveArgs {
  const uint32_t* code;      // table programs
  const int2* meta;          // [program] (code offset, length), in level order
  const int32_t* wcol;       // [program] its column; NULL: its number
  const uint8_t* kind;       // [program] kCol*
  const uint8_t* only;       // [program] counts only where only_value stands; NULL: all do
  uint8_t only_value;
  const int32_t* level_end;  // programs of level L end at level_end[L]
  int32_t n_levels;
  const ColStat* cst;        // [column] statistics of the rows done (FP64), or
  const unsigned long long* fnan;  // [column] first NaN row (double-float), of `rows` done
  int64_t rows;
  uint8_t* live;             // [column] out
};
bool launch_live_columns(const LiveArgs& a, cudaStream_t st);

// `list` (may be NULL) maps grid positions to candidates: candidate = list[cand0 + i].
// cst (may be NULL; one-column programs): column statistics of every
// written column, merged into cst[pc[c].a_col] (zeroed before the launch).
__global__ void plain_eval_kernel(DevBatch b, DevData ds, const PlainCand* pc, const int32_t* list, int cand0,
                                  double* A, uint32_t* status, ColStat* cst, EvalRows rows);
// colmap (may be NULL): factor column j of candidate c is column
// colmap[pc[c].a_col + j] of A (a shared factor table) instead of
// column pc[c].a_col + j.
// Column bucket of a QR launch for k + 1 columns (its widest sets the scratch).
int plain_qr_bucket(int cols);
// chained: as launch_next.  One block per candidate of the launch (the whole factorisation in one
// launch; QSUM order, the bits of launch_qr_chunked; qr_small.cu); max_cols
// bounds k + 1.
bool launch_plain_qr(int max_cols, int grid, int sm_count, cudaStream_t st, DevBatch b, DevData ds,
                     const PlainCand* pc, const int32_t* list, int cand0, const double* A, double* M, double* coefs,
                     rrg_result* res, uint32_t* status, const int32_t* colmap,
                     bool chained = false);
// Squared residual of the rebuilt sum of the candidates list[cand0 .. cand0 +
// n_cand) per chunk of RR_CHUNK rows: partial[c * chunks + chunk].  dcount (may
// be NULL): list positions at or beyond *dcount do nothing (a list whose length
// the device decided).
bool launch_plain_resid(DevBatch b, const DevData& ds, const PlainCand* pc, const int32_t* list, int cand0, int n_cand,
                        const double* A, const double* coefs, double* partial, const int32_t* colmap,
                        const int32_t* dcount, int sm_count, cudaStream_t st,
                        bool chained = false);
// partial[c * nb + j]: per-candidate squared-residual partial sums; when
// sse_direct is given and sse_direct[c] >= 0 (or NaN) it is the SSE itself.
__global__ void finalize_kernel(DevBatch b, DevData ds, const int32_t* list, int cand0, int cand1,
                                const double* partial, int nb, const double* coefs, rrg_result* res,
                                uint32_t flags_or, const double* sse_direct, const int32_t* dcount = nullptr);

__global__ void clear_results_kernel(const int32_t* list, int n, rrg_result* res, const int32_t* dcount = nullptr);

// Column statistics of an FP64 table: flags gathered by plain_eval_kernel, for
// deciding the column-pivoted QR's outcome on non-finite data without running
// it, and the column's sums of squares in QSUM order (launch_col_sums, where
// the chunked QR reads the column).
struct ColStat {
  uint32_t flags;   // kCs* bits
  uint32_t ticket;  // row chunks of the sums that are done
  double sumsq;     // over all rows
  double tailsq;    // over the rows after the first
};
constexpr uint32_t kCsNaN = 1;   // a NaN value: the column's norm is NaN
constexpr uint32_t kCsBig = 2;   // an infinite value or one whose square overflows
constexpr uint32_t kCsStop = 8;  // a NaN at row kStopRow or later: the remaining rows may be left out
// From this row on a NaN decides what a factor column can do in any refit:
// its rows up to the deepest pivot row are then all evaluated.
constexpr int64_t kStopRow = 128;
constexpr uint32_t kCsTail = 4;  // a row after the first with |value| > 1e-150 or non-finite
// The listed tuned candidates whose QR result is certain to be all-NaN
// coefficients at full rank (the fitness sentinel): that result is written,
// pc[c].pad = 1 (the QR and residual kernels skip it) and *decided counts it.
// sums: launch_col_sums has formed the listed candidates' columns' sums.
// gpart: nan_gram_bytes(n, cnt) bytes.  dcount as above.
size_t nan_gram_bytes(int64_t n, int cnt);
bool launch_nan_settle(const DevBatch& b, const DevData& ds, const int32_t* list, int cnt, PlainCand* pc,
                       const int32_t* colmap, const ColStat* cs, bool sums, const double* T, double* gpart,
                       double* coefs, rrg_result* res, uint32_t* decided, const int32_t* dcount, cudaStream_t st,
                       int64_t* launches);
// Before a table's evaluation: the listed results and the columns' statistics to zero.
bool launch_table_begin(const int32_t* list, int n, rrg_result* res, const int32_t* slots, int n_slots, ColStat* cst,
                        cudaStream_t st);
// Table columns listed in cols[0 .. *count) (one-column programs, pc[c].a_col
// = the column), with their column statistics into cst: a persistent grid of
// any size walks (column, row block) items, each column split into
// min(max_nbc, ceil(gridDim.x / count)) row blocks.  The values and
// statistics are those of plain_eval_kernel's one-column form.
__global__ void table_eval_list_kernel(DevBatch b, DevData ds, const PlainCand* pc, const int32_t* cols,
                                       const int32_t* count, int min_nbc, int max_nbc, double* A, uint32_t* status,
                                       ColStat* cst, EvalRows rows);

size_t plain_eval_smem(int levels = RRG_MAX_STACK, int words = kMaxCodeSmem);

}  // namespace rrd
