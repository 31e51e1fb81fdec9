// Column-pivoted QR least squares of the plain FP64 path for datasets of one
// chunk of rows (and for the allocation-free entry), one block per candidate:
// the factorisation of ColPivHouseholderQR::computeInPlace
// (eigen/Eigen/src/QR/ColPivHouseholderQR.h:482-575) on [factors | 1 | y], its
// least-squares solve (:577-608), with makeHouseholder /
// applyHouseholderOnTheLeft semantics (eigen/Eigen/src/Householder/Householder.h:67-133)
// and every sum in the QSUM order of csrc/common/rr_sum.h, bit for bit what
// qr_chunk.cu's passes give.
//
// At a few hundred rows the folds of the sums, the scalar work of a step and
// the waits between threads cost more than the rows do.  So a block has W = 1,
// 2, 4 or 8 warps and a warp carries 8 / W of QSUM's eight 32-lane groups: with
// one warp nothing waits for another.  The 8 / W groups of W columns are folded
// together (9 additions a warp for 8 sums, not 40); the scalars of a step (row
// kk, down-dating, back substitution) are one lane a column, each warp for
// itself; quotients and roots run on the integer pipes (fp64_int.h); the
// working columns stay in shared memory where they fit; the last step updates
// nothing, and the cut of the rank ends the factorisation.  GB300, the phase,
// against 256 threads a candidate with the scalars on one thread and the columns
// in device memory: 3190 candidates of 3 to 8 columns at 60 rows 0.52 -> 0.19 ms,
// at 569 0.66 -> 0.30, at 2500 1.74 -> 1.61, at 16384 (device memory) 9.1 -> 8.9;
// one candidate at 150 rows 43 -> 33 us.  Bound by the FP64 pipe from a few
// hundred rows up (44 instructions a warp and 32 rows at five columns: 0.17 ms
// at 569), below by the chain of dependent sums and scalars of each step.
#include <algorithm>
#include <cfloat>
#include <cstdint>
#include <type_traits>

#include "../common/fp64_int.h"
#include "../common/rr_sum.h"
#include "common.cuh"
#include "plain.cuh"
#include "qr_ops.cuh"
#include "reduce.cuh"

namespace rrd {

namespace {

constexpr double kDowndateThr = 1.4901161193847656e-08;  // sqrt(DBL_EPSILON)
constexpr int kRed = 9;                                  // doubles of a column's group sums (8, and 1 against bank conflicts)
constexpr size_t kSmemMax = 227 * 1024;
constexpr int kWarpsSm = 24;  // resident warps the registers allow

// Doubles of a block's shared state for up to mc columns (k + 1): group sums
// (two buffers), R by (step, column), and for each warp the norms, the sums and
// the columns' order.
__host__ __device__ constexpr int state_doubles(int W, int mc) {
  return 2 * kRed * mc + mc * (mc - 1) + W * (3 * mc + mc);
}

template <int W>
__device__ __forceinline__ void block_wait() {
  if (W == 1) __syncwarp();
  else __syncthreads();
}

// Group sums' storage and place in the block.
struct Sums {
  double* red;
  int mc, buf, lane, warp;
};

// out[q] = QSUM of term(q, row, .) over the rows [start, n), q < cnt, in every
// warp (start < n).  Ends with the columns' earlier stores visible to the block.
template <int W, class Row, class Term>
__device__ __forceinline__ void qsums(Sums& s, Row start, Row n, int cnt, double* out, Term term) {
  constexpr int G = 8 / W;
  for (Row c0 = start & ~(Row)(RR_CHUNK - 1); c0 < n; c0 += RR_CHUNK) {
    const Row lo = start > c0 ? start : c0, hi = n - c0 > RR_CHUNK ? c0 + RR_CHUNK : n;
    double* rd = s.red + s.buf * kRed * s.mc;
    s.buf ^= 1;
    for (int q0 = 0; q0 < cnt; q0 += W) {
      double acc[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = 0.0;
#pragma unroll(W == 8 ? 2 : 1)
      for (Row rb = lo & ~(Row)255; rb < hi; rb += 256) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const Row r = rb + 32 * (s.warp * G + g) + s.lane;
          if (r >= lo && r < hi) {
#pragma unroll
            for (int q = 0; q < W; ++q)
              if (q0 + q < cnt) acc[q * G + g] = term(q0 + q, r, acc[q * G + g]);
          }
        }
      }
      if (W > 1 && cnt - q0 == 1) {
        double one[G];
#pragma unroll
        for (int g = 0; g < G; ++g) one[g] = acc[g];
        const double v = warp_sum_many<G>(one);
        if ((s.lane & (32 / G - 1)) == 0) rd[q0 * kRed + s.warp * G + s.lane / (32 / G)] = v;
      } else {
        const double v = warp_sum_many<8>(acc);
        const int q = (s.lane >> 2) / G, g = (s.lane >> 2) % G;
        if ((s.lane & 3) == 0 && q0 + q < cnt) rd[(q0 + q) * kRed + s.warp * G + g] = v;
      }
    }
    block_wait<W>();
    for (int p = s.lane; p < cnt; p += 32) {
      // lane sums start from +0, so no total is -0: adding to 0, and the
      // totals of groups without a row, leave the bits as they are
      double v = rd[p * kRed];
#pragma unroll
      for (int i = 1; i < 8; ++i)
        if (32 * i < hi - c0) v = __dadd_rn(v, rd[p * kRed + i]);
      out[p] = c0 <= start ? v : __dadd_rn(out[p], v);
    }
    __syncwarp();
  }
}

template <int W, bool SMEM>
__global__ void __launch_bounds__(32 * W, kWarpsSm / W)
    qr_small_kernel(DevBatch b, DevData ds, const PlainCand* pc, const int32_t* list, int cand0, const double* A,
                    double* M, double* coefs, rrg_result* res, uint32_t* status, const int32_t* colmap, int mc) {
  constexpr int G = 8 / W;
  after_previous();
  using Row = typename std::conditional<SMEM, int, int64_t>::type;  // a column in shared memory has few rows
  extern __shared__ double smem[];
  const int c = list ? list[cand0 + blockIdx.x] : cand0 + blockIdx.x;
  if (b.cands[c].mode != RRG_TUNED || (pc[c].pad & 1)) return;  // pad bit 0: outcome already written
  const int k = pc[c].k;
  if (k + 1 > mc || k > RRG_MAX_TERMS) {
    if (threadIdx.x == 0) atomicOr(status, ST_TOO_LARGE);
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Row n = (Row)ds.n;
  Sums sm{smem, mc, 0, lane, warp};
  double* R = smem + 2 * kRed * mc;
  double* nupd = R + mc * (mc - 1) + warp * 4 * mc;  // by position, as ndir and tot
  double* ndir = nupd + mc;
  double* tot = ndir + mc;
  int32_t* pos = reinterpret_cast<int32_t*>(tot + mc);  // position -> column
  int32_t* rec = pos + mc;                              // positions whose norm is taken anew
  double* cols = SMEM ? smem + state_doubles(W, mc) : M + pc[c].m_col * ds.n_pad;
  const int64_t ld = SMEM ? ds.n : ds.n_pad;
  auto col = [&](int p) { return cols + pos[p] * ld; };
  auto rows_of = [&](Row start, auto f) {  // this thread's rows of [start, n), 8 / W at a time
    for (Row rb = start & ~(Row)255; rb < n; rb += 256) {
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const Row r = rb + 32 * (warp * G + g) + lane;
        if (r >= start && r < n) f(r);
      }
    }
  };

  for (int j = lane; j <= k; j += 32) pos[j] = j;
  for (int j = 0; j <= k; ++j) {
    double* dst = cols + j * ld;
    const double* src = j < k - 1 ? factor_column(A, ds.n_pad, pc[c].a_col, j, colmap) : ds.y64;
    if (j == k - 1) rows_of(0, [&](Row r) { dst[r] = 1.0; });
    else rows_of(0, [&](Row r) { dst[r] = src[r]; });
  }
  qsums<W, Row>(sm, 0, n, k, tot, [&](int q, Row r, double a) {
    const double x = cols[q * ld + r];
    return __fma_rn(x, x, a);
  });
  for (int j = lane; j < k; j += 32) nupd[j] = ndir[j] = fi_sqrt(tot[j]);
  __syncwarp();
  double maxn = nupd[0];
  for (int j = 1; j < k; ++j)
    if (fi_lt(maxn, nupd[j])) maxn = nupd[j];
  const double me = __dmul_rn(maxn, DBL_EPSILON);
  const double thr_helper = fi_div(__dmul_rn(me, me), (double)n);
  const int size = n < k ? (int)n : k;
  int rank = size;

  for (int kk = 0; kk < size; ++kk) {
    int big = kk;
    double bign = nupd[kk];
    for (int j = kk + 1; j < k; ++j)
      if (fi_lt(bign, nupd[j])) {
        bign = nupd[j];
        big = j;
      }
    if (fi_lt(__dmul_rn(bign, bign), __dmul_rn(thr_helper, (double)(n - kk)))) {
      rank = kk;
      break;
    }
    __syncwarp();
    if (lane == 0 && big != kk) {
      nupd[big] = nupd[kk];
      nupd[kk] = bign;
      const double t = ndir[big];
      ndir[big] = ndir[kk];
      ndir[kk] = t;
      const int32_t p = pos[big];
      pos[big] = pos[kk];
      pos[kk] = p;
    }
    __syncwarp();
    double* v = col(kk);
    double tail = 0.0;
    if (n - kk > 1) {
      qsums<W, Row>(sm, kk + 1, n, 1, tot, [&](int, Row r, double a) { return __fma_rn(v[r], v[r], a); });
      tail = tot[0];
      __syncwarp();
    } else {
      block_wait<W>();
    }
    double tau = 0.0, beta = v[kk];
    if (!(tail <= DBL_MIN)) {
      const double c0 = beta;
      beta = fi_sqrt(__dadd_rn(__dmul_rn(c0, c0), tail));
      if (c0 >= 0.0) beta = -beta;
      const fi_divisor rden = fi_divisor_of(__dsub_rn(c0, beta));
      rows_of(kk + 1, [&](Row r) { v[r] = fi_div_by(v[r], &rden); });
      tau = fi_div(__dsub_rn(beta, c0), beta);
    }
    if (threadIdx.x == 0) R[kk * mc + pos[kk]] = beta;
    const int cnt = k - kk;  // columns right of the pivot, y the last
    const bool apply = n - kk > 1 && !(tau == 0.0);
    if (apply)
      qsums<W, Row>(sm, kk + 1, n, cnt, tot, [&](int q, Row r, double a) { return __fma_rn(v[r], col(kk + 1 + q)[r], a); });
    // row kk, and the norms of what is left (LAWN 176, ColPivHouseholderQR.h:549-572)
    int nrec = 0;
    for (int p0 = 0; p0 < cnt; p0 += 32) {
      const int p = p0 + lane, j = kk + 1 + p;
      bool again = false;
      if (p < cnt) {
        double q = col(j)[kk];
        if (apply) {
          const double t = __dadd_rn(tot[p], q);
          tot[p] = t;
          q = __dsub_rn(q, __dmul_rn(tau, t));
        } else if (n - kk == 1) {
          q = __dmul_rn(q, __dsub_rn(1.0, tau));
        }
        if (warp == 0) R[kk * mc + pos[j]] = q;
        if (j < k && kk + 1 < size && nupd[j] != 0.0) {
          double temp = fi_div(fabs(q), nupd[j]);
          temp = __dmul_rn(__dadd_rn(1.0, temp), __dsub_rn(1.0, temp));
          temp = temp < 0.0 ? 0.0 : temp;
          const double ratio = fi_div(nupd[j], ndir[j]);
          again = __dmul_rn(temp, __dmul_rn(ratio, ratio)) <= kDowndateThr;
          if (!again) nupd[j] = __dmul_rn(nupd[j], fi_sqrt(temp));
        }
      }
      const uint32_t m = __ballot_sync(0xffffffffu, again);
      if (again) rec[nrec + __popc(m & ((1u << lane) - 1))] = j;
      nrec += __popc(m);
    }
    __syncwarp();
    if (kk + 1 == size) break;
    if (apply) {
      for (Row rb = (kk + 1) & ~255; rb < n; rb += 256) {
        double tv[G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const Row r = rb + 32 * (warp * G + g) + lane;
          tv[g] = r > kk && r < n ? -__dmul_rn(tau, v[r]) : 0.0;
        }
#pragma unroll(W == 8 ? 4 : 1)
        for (int p = 0; p < cnt; ++p) {
          double* a = col(kk + 1 + p);
          const double t = tot[p];
#pragma unroll
          for (int g = 0; g < G; ++g) {
            const Row r = rb + 32 * (warp * G + g) + lane;
            if (r > kk && r < n) a[r] = __fma_rn(tv[g], t, a[r]);
          }
        }
      }
      __syncwarp();
    }
    if (nrec > 0) {
      qsums<W, Row>(sm, kk + 1, n, nrec, tot, [&](int q, Row r, double a) {
        const double x = col(rec[q])[r];
        return __fma_rn(x, x, a);
      });
      for (int q = lane; q < nrec; q += 32) nupd[rec[q]] = ndir[rec[q]] = fi_sqrt(tot[q]);
      __syncwarp();
    }
  }
  if (warp != 0) return;
  // R c = Q'y by columns; coefficients beyond the rank are zero
  __syncwarp();
  for (int i = lane; i < rank; i += 32) tot[i] = R[i * mc + k];
  __syncwarp();
  for (int kk = rank - 1; kk >= 0; --kk) {
    const double x = fi_div(tot[kk], R[kk * mc + pos[kk]]);
    __syncwarp();
    if (lane == 0) tot[kk] = x;
    for (int i = lane; i < kk; i += 32) tot[i] = __dsub_rn(tot[i], __dmul_rn(x, R[i * mc + pos[kk]]));
    __syncwarp();
  }
  double* out = coefs + b.cands[c].coef_offset;
  for (int i = lane; i < k; i += 32) out[pos[i]] = i < rank ? tot[i] : 0.0;
  if (lane == 0) res[c].rank = rank;
}

template <int W, bool SMEM>
bool launch_w(size_t smem, int mc, int grid, cudaStream_t st, DevBatch b, DevData ds, const PlainCand* pc,
              const int32_t* list, int cand0, const double* A, double* M, double* coefs, rrg_result* res,
              uint32_t* status, const int32_t* colmap, bool chained) {
  if (smem > 48 * 1024 && cudaFuncSetAttribute(qr_small_kernel<W, SMEM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)kSmemMax) != cudaSuccess)
    return false;
  return launch_next(chained, qr_small_kernel<W, SMEM>, dim3(grid), 32 * W, smem, st, b, ds, pc, list, cand0, A, M, coefs, res,
                     status, colmap, mc) &&
         launch_ok("launch_plain_qr");
}

}  // namespace

bool launch_plain_qr(int max_cols, int grid, int sm_count, cudaStream_t st, DevBatch b, DevData ds,
                     const PlainCand* pc, const int32_t* list, int cand0, const double* A, double* M, double* coefs,
                     rrg_result* res, uint32_t* status, const int32_t* colmap, bool chained) {
  if (grid <= 0) return true;
  // Working columns in shared memory where one block's fit.  Then as few warps
  // a candidate as still give every SM 8 warps, counted over the launch: warps
  // beyond that only repeat the scalars (3190 candidates at 569 rows: 0.41 ms
  // for 4 warps an SM, 0.30 for 8, 0.41 for 16, 0.63 for 32; a lone candidate at
  // 150 rows 39 us with one warp, 33 with eight).
  auto bytes = [&](int W, bool in_smem) {
    return sizeof(double) * ((size_t)state_doubles(W, max_cols) + (in_smem ? (size_t)max_cols * (size_t)ds.n : 0));
  };
  const bool in_smem = bytes(8, true) <= kSmemMax;
  int W = in_smem ? 1 : 8;
  while (W < 8) {
    const int64_t per_sm = (int64_t)std::min<size_t>(kWarpsSm / W, (kSmemMax + 1024) / (bytes(W, true) + 1024));
    if (std::min<int64_t>(per_sm * sm_count, grid) * W >= 8 * (int64_t)sm_count) break;
    W *= 2;
  }
  const size_t sm = bytes(W, in_smem);
#define RRD_QR(W_, S_) \
  launch_w<W_, S_>(sm, max_cols, grid, st, b, ds, pc, list, cand0, A, M, coefs, res, status, colmap, chained)
  if (!in_smem) return RRD_QR(8, false);
  switch (W) {
    case 1: return RRD_QR(1, true);
    case 2: return RRD_QR(2, true);
    case 4: return RRD_QR(4, true);
    default: return RRD_QR(8, true);
  }
#undef RRD_QR
}

}  // namespace rrd
