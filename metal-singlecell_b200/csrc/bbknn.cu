// Batch-balanced kNN: metalsinglecell `neighbors.bbknn` (neighbors.py:491-559) and its trimming
// `_trim_graph` (neighbors.py:465-488), called by `pp.bbknn` (pp.py:809-833).
//
// Every cell gets, for every batch b, its kk_b = min(k, n_b) nearest cells of b (a cell of b finds
// itself at distance 0); the K = Σ kk_b entries of a cell are merged by (distance, index) and go
// through the same fuzzy simplicial set as pp.neighbors.  The reference scans each batch by brute
// force in FP32 (the n × n_b Gram matrix, neighbors.py:525-537); here the lists are exact:
//
//   layout   cells grouped by batch as the key side, batch b at packed rows [poff_b, poff_b + n_b)
//            (ascending cell index, each batch padded to SEG_PAD rows), and every cell once more
//            in a query region [P1, P1 + n) whose positions are never key columns, so the
//            candidate kernel's self-exclusion never drops a cell's own copy;
//   operands one centring (the mean of all cells) and one FP16 scale for both sides;
//   scan     per batch, one launch of the tensor-core candidate kernel in its row-list mode:
//            query tiles of 128 listed cells against the batch's key range, k' candidates per
//            cell and the k'-th value bounding every key left out;
//   re-rank  FP32 direct differences of the candidates, FP64 at the kk-th boundary, order by
//            (FP64 squared distance, index), and the same certificate as the self-kNN path; the
//            cells it cannot certify take an FP64 scan of the batch;
//   merge    every cell's K entries sorted by (float32 distance, index).
//
// Large inputs (BbPlan::ordered): the cells go into locality order first, queries and each batch's
// keys alike; a near pass scans every query tile's nearest key tile of each batch, and its radii give
// masks of the key tiles that can still matter (prune.cu), so that a query tile visits a few tiles
// of a batch instead of all.  All batches run in one launch per stage.  200,000 x 50, 8 batches, 3
// neighbours in each: the graph 35.3 ms batch by batch, 14.0 ordered.
//
// The distances graph drops the diagonal and every zero distance (neighbors.py:554-557); the
// trimming keeps an entry (i, j) of value v when v != 0, v >= θ_i and v >= θ_j, θ_i being the
// trim-th largest stored value of row i when the row stores more than `trim` entries, else 0.
#include <algorithm>
#include <cstdlib>

#include "kernels.cuh"
#include "msc_warpsort.cuh"

namespace msc {

namespace {

constexpr int BB_T = 256;
constexpr int BB_WARPS = BB_T / 32;
constexpr int BB_COLMEAN_NB = 256;

__host__ __device__ __forceinline__ int64_t bb_grid(int64_t units, int per_block) {
  return (units + per_block - 1) / per_block;
}

// ---- layout -------------------------------------------------------------------------------------

__global__ void bb_query_region_kernel(int64_t n, int64_t p1, int32_t* __restrict__ perm,
                                       int32_t* __restrict__ qmap) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    perm[p1 + i] = int32_t(i);
    qmap[i] = int32_t(p1 + i);
  }
}

__global__ void bb_flag_kernel(const int32_t* __restrict__ codes, int64_t n, int b,
                               int32_t* __restrict__ flag) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x)
    flag[i] = codes[i] == b ? 1 : 0;
}

// cells of batch b to [poff, poff + nb) in ascending cell order; a cell beyond the stated count
// (codes and counts that disagree) is not placed, so no write leaves the batch's rows
__global__ void bb_place_kernel(const int32_t* __restrict__ codes, int64_t n, int b,
                                const int64_t* __restrict__ S, int64_t poff, int64_t nb,
                                int32_t* __restrict__ perm) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    if (codes[i] != b) continue;
    const int64_t r = S[i];
    if (r < nb) perm[poff + r] = int32_t(i);
  }
}

// the same from the cells in locality order (positions j, cells gperm[j])
__global__ void bb_flag_order_kernel(const int32_t* __restrict__ codes,
                                     const int32_t* __restrict__ gperm, int64_t n, int b,
                                     int32_t* __restrict__ flag) {
  for (int64_t j = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; j < n;
       j += int64_t(gridDim.x) * blockDim.x)
    flag[j] = codes[gperm[j]] == b ? 1 : 0;
}
__global__ void bb_place_order_kernel(const int32_t* __restrict__ flag,
                                      const int32_t* __restrict__ gperm,
                                      const int32_t* __restrict__ gleaf, int64_t n,
                                      const int64_t* __restrict__ S, int64_t poff, int64_t nb,
                                      int32_t* __restrict__ perm, int32_t* __restrict__ leaf) {
  for (int64_t j = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; j < n;
       j += int64_t(gridDim.x) * blockDim.x) {
    const int64_t r = S[j];
    if (flag[j] && r < nb) {
      perm[poff + r] = gperm[j];
      leaf[poff + r] = gleaf[j];
    }
  }
}
__global__ void bb_query_order_kernel(const int32_t* __restrict__ gperm,
                                      const int32_t* __restrict__ gleaf, int64_t n, int64_t p1,
                                      int32_t* __restrict__ perm, int32_t* __restrict__ leaf,
                                      int32_t* __restrict__ qmap) {
  for (int64_t j = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; j < n;
       j += int64_t(gridDim.x) * blockDim.x) {
    perm[p1 + j] = gperm[j];
    leaf[p1 + j] = gleaf[j];
    qmap[j] = int32_t(p1 + j);
  }
}

// the batches of one launch
constexpr int BB_GROUP = 64;
struct BbBatches {
  int32_t poff[BB_GROUP], nb[BB_GROUP], kk[BB_GROUP], col0[BB_GROUP];
  int32_t start[BB_GROUP];      // of the batch's cells in the list in storage order
};

// batch-major items of a group: scan items (query rows of the list) and plan items (packed rows)
__global__ void bb_group_items_kernel(const BbBatches B, int nb, int64_t n, int64_t p1,
                                      WorkItem* __restrict__ items,
                                      WorkItem* __restrict__ pitems) {
  const int64_t nt = (n + QTILE - 1) / QTILE;
  for (int64_t x = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; x < nt * nb;
       x += int64_t(gridDim.x) * blockDim.x) {
    const int b = int(x / nt);
    const int64_t t = x - b * nt;
    WorkItem w;
    w.qrow0 = int32_t(t * QTILE);
    w.nq = int32_t(min64(QTILE, n - t * QTILE));
    w.key0 = B.poff[b];
    w.nkeys = B.nb[b];
    w.orig_off = 0;
    w.qorig0 = 0;
    w.pad0 = b;
    w.pad1 = 0;
    items[x] = w;
    w.qrow0 += int32_t(p1);
    pitems[x] = w;
  }
}

// The cells of every batch about as they are stored, batch b's from start[b] on, for the FP64 scans
// of a group: neighbouring rows share cache lines, which rows in locality order do not.  (59,948 x 25
// in BF16 with nearly every cell scanned: 114 ms in locality order, 100 so.)  Nothing to scan, nothing
// done.
__global__ void bb_store_order_kernel(const int32_t* __restrict__ codes, int64_t n,
                                      const BbBatches B, int nb, int first,
                                      const int32_t* __restrict__ nrows,
                                      int32_t* __restrict__ cursor, int32_t* __restrict__ list) {
  if (*nrows == 0) return;
  const int lane = lane_id();
  for (int64_t j0 = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) / 32 * 32; j0 < n;
       j0 += int64_t(gridDim.x) * blockDim.x) {          // warp-uniform
    const int64_t j = j0 + lane;
    int b = j < n ? codes[j] - first : -1;
    if (b < 0 || b >= nb) b = -1;
    const unsigned same = __match_any_sync(FULL, b);
    int at = 0;
    if (b >= 0 && lane == __ffs(same) - 1) at = atomicAdd(&cursor[b], __popc(same));
    at = __shfl_sync(FULL, at, __ffs(same) - 1) + __popc(same & ((1u << lane) - 1u));
    if (b >= 0 && at < B.nb[b]) list[B.start[b] + at] = int32_t(j);
  }
}

__global__ void bb_set_i32_kernel(int32_t* __restrict__ p, int32_t v) { *p = v; }

// query tiles of batch b: 128 listed cells each against the batch's keys
__global__ void bb_items_kernel(int64_t n, int64_t poff, int64_t nb, WorkItem* __restrict__ items) {
  const int64_t nt = (n + QTILE - 1) / QTILE;
  for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < nt;
       t += int64_t(gridDim.x) * blockDim.x) {
    WorkItem w;
    w.qrow0 = int32_t(t * QTILE);
    w.nq = int32_t(min64(QTILE, n - t * QTILE));
    w.key0 = int32_t(poff);
    w.nkeys = int32_t(nb);
    w.orig_off = 0;
    w.qorig0 = 0;
    w.pad0 = 0;
    w.pad1 = 0;
    items[t] = w;
  }
}

// ---- exact re-rank of one batch's candidates ----------------------------------------------------

__device__ __forceinline__ double bb_d2_f64(const float* xs, const float* __restrict__ y, int d) {
  double acc = 0.0;
  for (int t = 0; t < d; ++t) {
    const double df = double(xs[t]) - double(y[t]);
    acc += df * df;
  }
  return acc;
}
__device__ __forceinline__ float bb_d2_f32(const float* xs, const float* __restrict__ y, int d) {
  float acc = 0.f;
  for (int t = 0; t < d; ++t) {
    const float df = xs[t] - y[t];
    acc = fmaf(df, df, acc);
  }
  return acc;
}

// four lanes' shares of an FP32 squared distance (part = lane & 3 takes every fourth 8-byte pair, or
// every fourth element of a row that is not 8-byte aligned); any order of the sum stays within the
// (d+4)·2^-24 the windows assume
__device__ __forceinline__ float bb_part_d2_f32(const float* xs, const float* __restrict__ y,
                                                int d, int part) {
  float a0 = 0.f, a1 = 0.f;
  if ((reinterpret_cast<uintptr_t>(y) & 7) == 0) {
    const float2* y2 = reinterpret_cast<const float2*>(y);
    const float2* x2 = reinterpret_cast<const float2*>(xs);
    const int h = d >> 1;
    for (int t = part; t < h; t += 4) {
      const float2 u = y2[t], p = x2[t];
      const float e0 = p.x - u.x, e1 = p.y - u.y;
      a0 = fmaf(e0, e0, a0);
      a1 = fmaf(e1, e1, a1);
    }
    if ((d & 1) && part == 0) {
      const float e = xs[d - 1] - y[d - 1];
      a0 = fmaf(e, e, a0);
    }
  } else {
    for (int t = part; t < d; t += 4) {
      const float e = xs[t] - y[t];
      a0 = fmaf(e, e, a0);
    }
  }
  return a0 + a1;
}

// a warp's FP64 scan of keys perm[lo..hi) for cell i (xs: its row): the kk <= 128 nearest by
// (d², index) in top
__device__ __forceinline__ void bb_scan_keys(const float* __restrict__ X, int d, int64_t i,
                                             const int32_t* __restrict__ perm, int64_t lo,
                                             int64_t hi, int kk, float* xs, WarpTop128& top) {
  const int lane = lane_id();
  for (int t = lane; t < d; t += 32) xs[t] = X[i * d + t];
  __syncwarp();
  top.init();
  for (int64_t base = lo; base < hi; base += 32) {
    const int64_t jj = base + lane;
    double v = __longlong_as_double(0x7ff0000000000000ll);
    int vi = INT32_MAX;
    if (jj < hi) {
      const int32_t c = perm[jj];
      if (c >= 0) {
        v = bb_d2_f64(xs, X + int64_t(c) * d, d);
        vi = c;
      }
    }
    top.offer(v, vi, kk);
  }
}
// a cell's kk neighbours in a batch to oi / od (warp-collective)
__device__ __forceinline__ void bb_write_row(const WarpTop128& top, int64_t i, int kk, int32_t* oi,
                                             float* od) {
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const int r = s * 32 + lane_id();
    if (r < kk) {
      oi[r] = top.ai[s] == INT32_MAX ? int32_t(i) : top.ai[s];
      od[r] = __double2float_rn(sqrt(top.a[s]));
    }
  }
  __syncwarp();
}

// A block's FP64 scan of a batch for one cell: its warps take an eighth of the keys each and are
// merged (kk <= 32).  While there are no more cells to scan than blocks this is what the scans do: a
// lone cell is otherwise one warp's chain of FP64 sums over the whole batch.  56,723 x 50 with 23
// such cells 6.9 -> 4.3 ms, 54,089 x 7 with 41 3.8 -> 2.6.  The warps' lists take the place of their
// rows (xs): shared memory of their own would cost the scans of many cells L1, 2 to 4 %.
__device__ __forceinline__ void bb_scan_block(const float* __restrict__ X, int d, int64_t i,
                                              const int32_t* __restrict__ perm, int64_t nb, int kk,
                                              float (*xs)[MSC_MAX_D], int32_t* oi, float* od) {
  static_assert(sizeof(xs[0]) >= 32 * (sizeof(double) + sizeof(int)), "a list fits a row");
  const int lane = lane_id(), wib = warp_id();
  const int64_t per = (nb + BB_WARPS * 32 - 1) / (BB_WARPS * 32) * 32;
  WarpTop128 top;
  bb_scan_keys(X, d, i, perm, wib * per, min64(nb, (wib + 1) * per), kk, xs[wib], top);
  __syncwarp();                                          // the row is read
  reinterpret_cast<double*>(xs[wib])[lane] = top.a[0];
  reinterpret_cast<int*>(xs[wib])[64 + lane] = top.ai[0];
  __syncthreads();
  if (wib == 0) {
    for (int q = 1; q < BB_WARPS; ++q)
      top.offer(reinterpret_cast<const double*>(xs[q])[lane],
                reinterpret_cast<const int*>(xs[q])[64 + lane], kk);
    bb_write_row(top, i, kk, oi, od);
  }
}

// One warp per cell i: its k' candidates in batch b (original rows, -1 = none) → the kk nearest
// by (FP64 d², index) into columns [col0, col0 + kk) of row i; uncertified cells to fail_rows.
__global__ void __launch_bounds__(BB_T)
bb_rerank_kernel(const float* __restrict__ X, int d, int64_t n, int64_t p1,
                 const int32_t* __restrict__ cand_idx, const float* __restrict__ cand_thr,
                 int kprime, const QStat* __restrict__ qs, const KeyMax* __restrict__ km,
                 const Ctl* __restrict__ ctl, int prec, int kmma, int64_t nb, int kk, int K,
                 int col0, int32_t* __restrict__ knn_idx, float* __restrict__ knn_dist,
                 int32_t* __restrict__ fail_rows, int32_t* __restrict__ nfail,
                 int64_t* __restrict__ n_cert_out) {
  __shared__ __align__(16) float xs_all[BB_WARPS][MSC_MAX_D];
  const int lane = lane_id(), wib = warp_id();
  float* xs = xs_all[wib];
  const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  const KeyMax kmv = *km;
  const double f = op_scale(prec, ctl);
  const double f2 = f * f;
  const double delta = double(d + 4) * 0x1p-24;
  const double INF = __longlong_as_double(0x7ff0000000000000ll);
  int64_t n_cert = 0;
  for (int64_t i = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5; i < n; i += nwarps) {
    for (int t = lane; t < d; t += 32) xs[t] = X[i * d + t];
    __syncwarp();
    int c0 = lane < kprime ? cand_idx[i * kprime + lane] : -1;
    int c1 = lane + 32 < kprime ? cand_idx[i * kprime + lane + 32] : -1;
    double v0 = c0 >= 0 ? double(bb_d2_f32(xs, X + int64_t(c0) * d, d)) : INF;
    double v1 = c1 >= 0 ? double(bb_d2_f32(xs, X + int64_t(c1) * d, d)) : INF;
    int i0 = c0 >= 0 ? c0 : INT32_MAX, i1 = c1 >= 0 ? c1 : INT32_MAX;
    warp_sort64_d(v0, i0, v1, i1);
    const double B = __shfl_sync(FULL, kk - 1 < 32 ? v0 : v1, (kk - 1) & 31);
    // FP64 for the window of FP32 values within B·(1+3δ) and the rounding of subnormal sums
    const double lim = B * (1.0 + 3.0 * delta) + 2.0 * F32_SQ_FLOOR;
    const bool w0 = i0 != INT32_MAX && v0 <= lim;
    const bool w1 = i1 != INT32_MAX && v1 <= lim;
    double g0 = w0 ? bb_d2_f64(xs, X + int64_t(i0) * d, d) : INF;
    double g1 = w1 ? bb_d2_f64(xs, X + int64_t(i1) * d, d) : INF;
    int h0 = w0 ? i0 : INT32_MAX, h1 = w1 ? i1 : INT32_MAX;
    warp_sort64_d(g0, h0, g1, h1);
    const double Dk = __shfl_sync(FULL, kk - 1 < 32 ? g0 : g1, (kk - 1) & 31);
    bool cert;
    if (nb <= kprime) {
      cert = true;                                     // every key of the batch is a candidate
    } else {
      const QStat q = qs[p1 + i];
      const double eps = cert_eps(q, kmv, prec, kmma, d);
      cert = f2 * Dk < q.sq + double(cand_thr[i]) - eps;
    }
    int32_t* oi = knn_idx + i * K + col0;
    float* od = knn_dist + i * K + col0;
    if (lane < kk) {
      oi[lane] = h0 == INT32_MAX ? int32_t(i) : h0;
      od[lane] = __double2float_rn(sqrt(g0));
    }
    if (lane + 32 < kk) {
      oi[lane + 32] = h1 == INT32_MAX ? int32_t(i) : h1;
      od[lane + 32] = __double2float_rn(sqrt(g1));
    }
    if (lane == 0) {
      if (cert) ++n_cert;
      else fail_rows[atomicAdd(nfail, 1)] = int32_t(i);
    }
    __syncwarp();
  }
  if (lane == 0 && n_cert)
    atomicAdd(reinterpret_cast<unsigned long long*>(n_cert_out), (unsigned long long)n_cert);
}

// One warp per cell of the order and group of batches: its k' <= 32 candidates of each batch, as in
// rerank.cu: FP32 distances with four lanes a candidate, the kk-th from a sort of the values alone,
// FP64 for the few within its rounding bound, placed by counting.  (The kernel above reads a
// candidate's row with one lane and sorts 64 FP64 pairs twice: 7.7 ms for 8 batches of 200,000
// cells, 2.7 here.)  Cells it cannot certify, or with more than 32 candidates inside the bound
// or NaN distances, are listed for the FP64 scan.
__global__ void __launch_bounds__(BB_T)
bb_group_rerank_kernel(const float* __restrict__ X, int d, int64_t n, int64_t p1,
                       const int32_t* __restrict__ perm, const BbBatches B, int nb,
                       const int32_t* __restrict__ cand_idx, const float* __restrict__ cand_thr,
                       int kprime, const QStat* __restrict__ qs, const KeyMax* __restrict__ km,
                       const Ctl* __restrict__ ctl, int prec, int kmma, int K,
                       int32_t* __restrict__ knn_idx, float* __restrict__ knn_dist,
                       int32_t* __restrict__ fail_rows, int32_t* __restrict__ fail_bat,
                       int32_t* __restrict__ nfail, int64_t* __restrict__ n_cert_out) {
  __shared__ __align__(16) float xs_all[BB_WARPS][MSC_MAX_D];
  __shared__ int win_all[BB_WARPS][32];
  const int lane = lane_id(), wib = warp_id();
  float* xs = xs_all[wib];
  int* win = win_all[wib];
  const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  const KeyMax kmv = *km;
  const double f = op_scale(prec, ctl);
  const double f2 = f * f;
  const double delta = double(d + 4) * 0x1p-24;
  const double INF = __longlong_as_double(0x7ff0000000000000ll);
  const unsigned lt = (1u << lane) - 1u;
  int64_t n_cert = 0;
  for (int64_t j = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5; j < n; j += nwarps) {
    const int64_t i = perm[p1 + j];
    __syncwarp();
    for (int t = lane; t < d; t += 32) xs[t] = X[i * d + t];
    __syncwarp();
    const QStat q = qs[p1 + j];
    const double eps = cert_eps(q, kmv, prec, kmma, d);
    for (int b = 0; b < nb; ++b) {
      const int kk = B.kk[b];
      const int c = lane < kprime ? cand_idx[(i * nb + b) * kprime + lane] : -1;
      float e = F_INF;
      for (int r = 0; r < kprime; r += 8) {              // eight candidates, four lanes each
        const int s = r + (lane >> 2);
        const int cid = __shfl_sync(FULL, c, s & 31);
        const bool have = s < kprime && cid >= 0;
        float v = have ? bb_part_d2_f32(xs, X + int64_t(cid) * d, d, lane & 3) : 0.f;
        v += __shfl_xor_sync(FULL, v, 1);
        v += __shfl_xor_sync(FULL, v, 2);
        if (!have) v = F_INF;
        const float got = __shfl_sync(FULL, v, ((lane - r) & 7) * 4);
        if (lane >= r && lane < r + 8) e = got;
      }
      bool ok = !__any_sync(FULL, isnan(e));
      float sv = e;
      warp_sort32_f(sv);
      const double lim = double(__shfl_sync(FULL, sv, kk - 1)) * (1.0 + 3.0 * delta) + 2.0 * F32_SQ_FLOOR;
      const bool in = c >= 0 && double(e) <= lim;
      const unsigned m = __ballot_sync(FULL, in);
      const int nw = __popc(m);
      ok = ok && nw >= kk;
      if (ok) {                                          // warp-uniform
        if (in) win[__popc(m & lt)] = c;
        __syncwarp();
        const int id = lane < nw ? win[lane] : INT32_MAX;
        const double g = lane < nw ? bb_d2_f64(xs, X + int64_t(id) * d, d) : INF;
        int rank = 0;
        for (int x = 0; x < nw; ++x) {
          const double og = __shfl_sync(FULL, g, x);
          const int oi = __shfl_sync(FULL, id, x);
          rank += dless(og, oi, g, id);
        }
        // every key outside the list has an approximate value at or above T
        const double T = double(cand_thr[b * n + i]);
        const bool mine = lane < nw && rank == kk - 1 &&
                          (B.nb[b] <= kprime || f2 * g < q.sq + T - eps);
        ok = __any_sync(FULL, mine);
        if (lane < nw && rank < kk) {
          knn_idx[i * K + B.col0[b] + rank] = id;
          knn_dist[i * K + B.col0[b] + rank] = __double2float_rn(sqrt(g));
        }
        __syncwarp();
      }
      if (lane == 0) {
        if (ok) {
          ++n_cert;
        } else {
          const int at = atomicAdd(nfail, 1);
          fail_rows[at] = int32_t(i);
          fail_bat[at] = b;
        }
      }
    }
  }
  if (lane == 0 && n_cert)
    atomicAdd(reinterpret_cast<unsigned long long*>(n_cert_out), (unsigned long long)n_cert);
}

// FP64 scan of the listed (cell, batch) pairs of a group: a warp each, or a block (bb_scan_block)
__global__ void __launch_bounds__(BB_T)
bb_group_scan_kernel(const float* __restrict__ X, int d, const int32_t* __restrict__ list,
                     const BbBatches B, const int32_t* __restrict__ rows,
                     const int32_t* __restrict__ bats, const int32_t* __restrict__ nrows, int K,
                     int32_t* __restrict__ knn_idx, float* __restrict__ knn_dist,
                     int64_t* __restrict__ n_scanned) {
  __shared__ __align__(16) float xs_all[BB_WARPS][MSC_MAX_D];
  const int lane = lane_id(), wib = warp_id();
  const int64_t count = *nrows;
  if (count <= gridDim.x) {
    if (blockIdx.x >= count) return;
    const int b = bats[blockIdx.x];
    const int64_t i = rows[blockIdx.x];
    bb_scan_block(X, d, i, list + B.start[b], B.nb[b], B.kk[b], xs_all,
                  knn_idx + i * K + B.col0[b], knn_dist + i * K + B.col0[b]);
    if (threadIdx.x == 0) atomicAdd(reinterpret_cast<unsigned long long*>(n_scanned), 1ull);
    return;
  }
  WarpTop128 top;
  const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  int64_t done = 0;
  for (int64_t w = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5; w < count;
       w += nwarps) {
    const int b = bats[w], kk = B.kk[b];
    const int64_t i = rows[w];
    bb_scan_keys(X, d, i, list + B.start[b], 0, B.nb[b], kk, xs_all[wib], top);
    bb_write_row(top, i, kk, knn_idx + i * K + B.col0[b], knn_dist + i * K + B.col0[b]);
    ++done;
  }
  if (lane == 0 && done)
    atomicAdd(reinterpret_cast<unsigned long long*>(n_scanned), (unsigned long long)done);
}

// FP64 scan of batch b for the listed cells (every cell when rows == nullptr): the kk (<= 128)
// nearest keys by (d², index) into columns [col0, col0 + kk)
__global__ void __launch_bounds__(BB_T)
bb_scan_kernel(const float* __restrict__ X, int d, int64_t n, const int32_t* __restrict__ perm,
               int64_t poff, int64_t nb, const int32_t* __restrict__ rows,
               const int32_t* __restrict__ nrows, int kk, int K, int col0,
               int32_t* __restrict__ knn_idx, float* __restrict__ knn_dist,
               int64_t* __restrict__ n_scanned) {
  __shared__ __align__(16) float xs_all[BB_WARPS][MSC_MAX_D];
  const int lane = lane_id(), wib = warp_id();
  const int64_t count = rows ? int64_t(*nrows) : n;
  if (rows && count <= gridDim.x && kk <= 32) {
    if (blockIdx.x >= count) return;
    const int64_t i = rows[blockIdx.x];
    bb_scan_block(X, d, i, perm + poff, nb, kk, xs_all, knn_idx + i * K + col0,
                  knn_dist + i * K + col0);
    if (threadIdx.x == 0) atomicAdd(reinterpret_cast<unsigned long long*>(n_scanned), 1ull);
    return;
  }
  const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  int64_t done = 0;
  for (int64_t w = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5; w < count;
       w += nwarps) {
    const int64_t i = rows ? int64_t(rows[w]) : w;
    WarpTop128 top;
    bb_scan_keys(X, d, i, perm + poff, 0, nb, kk, xs_all[wib], top);
    bb_write_row(top, i, kk, knn_idx + i * K + col0, knn_dist + i * K + col0);
    ++done;
  }
  if (lane == 0 && done)
    atomicAdd(reinterpret_cast<unsigned long long*>(n_scanned), (unsigned long long)done);
}

// every row's K (<= 128) entries in (float32 distance, index) order: each entry's rank is the
// number of entries before it
__global__ void __launch_bounds__(BB_T)
bb_merge_kernel(int64_t n, int K, int32_t* __restrict__ knn_idx, float* __restrict__ knn_dist) {
  __shared__ float dv_all[BB_WARPS][128];
  __shared__ int32_t iv_all[BB_WARPS][128];
  const int lane = lane_id(), wib = warp_id();
  float* dv = dv_all[wib];
  int32_t* iv = iv_all[wib];
  const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t i = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5; i < n; i += nwarps) {
    for (int e = lane; e < K; e += 32) {
      dv[e] = knn_dist[i * K + e];
      iv[e] = knn_idx[i * K + e];
    }
    __syncwarp();
    for (int e = lane; e < K; e += 32) {
      const float de = dv[e];
      const int32_t ie = iv[e];
      int r = 0;
      for (int g = 0; g < K; ++g)
        r += (dv[g] < de || (dv[g] == de && (iv[g] < ie || (iv[g] == ie && g < e)))) ? 1 : 0;
      knn_idx[i * K + r] = ie;
      knn_dist[i * K + r] = de;
    }
    __syncwarp();
  }
}

// ---- distances graph ---------------------------------------------------------------------------

__device__ __forceinline__ bool bb_dist_kept(int32_t j, float v, int64_t i) {
  return int64_t(j) != i && v != 0.f;
}

__global__ void bb_dist_count_kernel(const int32_t* __restrict__ idx, const float* __restrict__ dist,
                                     int64_t n, int K, int32_t* __restrict__ cnt) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    int c = 0;
    for (int e = 0; e < K; ++e) c += bb_dist_kept(idx[i * K + e], dist[i * K + e], i) ? 1 : 0;
    cnt[i] = c;
  }
}

// row i's kept entries in column order (the columns of a row are distinct)
__global__ void __launch_bounds__(BB_T)
bb_dist_fill_kernel(const int32_t* __restrict__ idx, const float* __restrict__ dist, int64_t n,
                    int K, const int64_t* __restrict__ indptr, int32_t* __restrict__ indices,
                    float* __restrict__ data) {
  __shared__ int32_t col_all[BB_WARPS][128];
  const int lane = lane_id(), wib = warp_id();
  int32_t* col = col_all[wib];
  const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t i = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5; i < n; i += nwarps) {
    for (int e = lane; e < K; e += 32) {
      const int32_t j = idx[i * K + e];
      col[e] = bb_dist_kept(j, dist[i * K + e], i) ? j : -1;
    }
    __syncwarp();
    const int64_t base = indptr[i];
    for (int e = lane; e < K; e += 32) {
      const int32_t j = col[e];
      if (j < 0) continue;
      int r = 0;
      for (int g = 0; g < K; ++g) r += (col[g] >= 0 && col[g] < j) ? 1 : 0;
      indices[base + r] = j;
      data[base + r] = dist[i * K + e];
    }
    __syncwarp();
  }
}

// ---- trimming ----------------------------------------------------------------------------------

// float -> unsigned with the same order (negative values below positive ones)
__device__ __forceinline__ uint32_t ord_key(float v) {
  const uint32_t b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float ord_val(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// θ_i = the trim-th largest stored value of row i when the row stores more than `trim` entries,
// else 0: the largest key t with #{v : key(v) >= t} >= trim, found bit by bit from the top
__global__ void __launch_bounds__(BB_T)
trim_theta_kernel(const int64_t* __restrict__ indptr, const float* __restrict__ data, int64_t n,
                  int trim, float* __restrict__ theta) {
  const int lane = lane_id();
  const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t i = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5; i < n; i += nwarps) {
    const int64_t a = indptr[i], b = indptr[i + 1];
    if (b - a <= trim) {
      if (lane == 0) theta[i] = 0.f;
      continue;
    }
    uint32_t t = 0;
    for (int bit = 31; bit >= 0; --bit) {
      const uint32_t test = t | (1u << bit);
      int64_t c = 0;
      for (int64_t e = a + lane; e < b; e += 32) c += ord_key(data[e]) >= test ? 1 : 0;
      for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(FULL, c, o);
      if (c >= trim) t = test;
    }
    if (lane == 0) theta[i] = ord_val(t);
  }
}

__device__ __forceinline__ bool trim_kept(float v, float ti, float tj) {
  return v != 0.f && v >= ti && v >= tj;
}

__global__ void trim_count_kernel(const int64_t* __restrict__ indptr,
                                  const int32_t* __restrict__ indices,
                                  const float* __restrict__ data, int64_t n,
                                  const float* __restrict__ theta, int32_t* __restrict__ cnt) {
  // a warp per row: a thread per row read its row entry by entry, 0.31 ms for 7 M entries
  const int lane = lane_id();
  const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t i = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5; i < n; i += nwarps) {
    const float ti = theta[i];
    const int64_t b = indptr[i + 1];
    int c = 0;
    for (int64_t e = indptr[i] + lane; e < b; e += 32)
      c += trim_kept(data[e], ti, theta[indices[e]]) ? 1 : 0;
    c = __reduce_add_sync(FULL, c);
    if (lane == 0) cnt[i] = c;
  }
}

// the kept entries of each row, in their stored order
__global__ void __launch_bounds__(BB_T)
trim_fill_kernel(const int64_t* __restrict__ indptr, const int32_t* __restrict__ indices,
                 const float* __restrict__ data, int64_t n, const float* __restrict__ theta,
                 const int64_t* __restrict__ out_ptr, int32_t* __restrict__ out_idx,
                 float* __restrict__ out_data) {
  const int lane = lane_id();
  const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t i = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5; i < n; i += nwarps) {
    const int64_t a = indptr[i], b = indptr[i + 1];
    const float ti = theta[i];
    int64_t o = out_ptr[i];
    for (int64_t e0 = a; e0 < b; e0 += 32) {
      const int64_t e = e0 + lane;
      bool keep = false;
      int32_t j = 0;
      float v = 0.f;
      if (e < b) {
        j = indices[e];
        v = data[e];
        keep = trim_kept(v, ti, theta[j]);
      }
      const unsigned m = __ballot_sync(FULL, keep);
      if (keep) {
        const int64_t at = o + __popc(m & ((1u << lane) - 1u));
        out_idx[at] = j;
        out_data[at] = v;
      }
      o += __popc(m);
    }
  }
}

int grid_for(int64_t units, int per_block) {
  return int(std::max<int64_t>(1, std::min<int64_t>(bb_grid(units, per_block),
                                                    int64_t(num_sms()) * 16)));
}

}  // namespace

// ---- host side ---------------------------------------------------------------------------------

namespace {
constexpr int64_t BB_ORDER_MIN = 32768;
constexpr int BB_ORDER_LEAF = 256;
}  // namespace

BbPlan bb_plan(int64_t n, int d, const int64_t* counts, int nb, int kwb, int prec) {
  BbPlan P;
  P.n = n;
  P.d = d;
  P.nb = nb;
  P.kwb = kwb;
  P.prec = prec;
  P.K = 0;
  P.kk_max = 0;
  P.p1 = 0;
  P.max_nb = 0;
  for (int b = 0; b < nb; ++b) {
    const int kk = int(std::min<int64_t>(kwb, counts[b]));
    P.K += kk;
    P.kk_max = std::max(P.kk_max, kk);
    P.p1 += round_up(std::max<int64_t>(counts[b], 1), SEG_PAD);
    P.max_nb = std::max(P.max_nb, counts[b]);
  }
  P.npk = P.p1 + round_up(n, QTILE);
  // candidates: the one-term tensor-core scan with the self-kNN path's over-fetch for k = kk+1
  P.candidates = P.kk_max + 1 <= 64 && prec != PREC_FP32 && d <= MSC_MAX_D;
  P.kprime = 0;
  if (P.candidates) {
    // over-fetch: the certificate compares the kk-th neighbour with the k'-th candidate (the self
    // path's k' = 48 is sized for the 15th neighbour), and a cell that it cannot certify takes an
    // FP64 scan of the batch.  24 candidates save 6 to 10 % against 32 where no cell fails (8 batches
    // of 200,000 x 50, FP16: 13.7 and 14.7 ms).  For up to six neighbours they leave none to some
    // tens of cells that 32 would not; for more, or with BF16 operands, they left thousands
    // (60,000 x 50 BF16 146 ms against 91; 132,000 x 50 FP16 with 13 neighbours 19.0 against 15.1).
    // The three-term split left none at 24.
    const bool few = prec == PREC_FP16 && P.kk_max <= 6;
    P.kprime = prec == PREC_BF16X3 ? std::min(64, std::max(24, P.kk_max + 9))
                                   : std::min(64, std::max(few ? 24 : 32, P.kk_max + 16));
    P.L = op_layout(prec, d);
    P.cfg = tc_default_config(prec, d, P.kprime);
    if (P.cfg.pair || !tc_config_ok(P.cfg, P.L.kp, P.kprime)) P.candidates = false;
  }
  P.ntiles = ceil_div(n, QTILE);
  // the ordered scan: lists the group re-rank takes, 256-key tiles, and enough cells that the order
  // and the plan cost less than the tiles they save.  Batch by batch the scan is a launch per stage
  // and batch, so the line lies lower the more batches there are.  ms batch by batch / ordered:
  //            clustered data                  Gaussian data (nothing to prune)
  //   cells    2 batches    8                  2            8
  //   33,000   1.62 / 2.71  3.42 / 3.23        1.62 / 2.68  3.48 / 3.91
  //   45,000   2.65 / 2.91  5.43 / 3.88        2.65 / 3.32  5.45 / 5.17
  //   60,000   3.73 / 3.25  7.43 / 4.70        3.73 / 4.34  7.46 / 6.88
  // The line is where clustered data, the usual, is even (4 batches: about 38,000).
  // MSC_B200_BB_ORDER=<cells> moves it (tests; 0: always, negative: never).
  int64_t least = std::max<int64_t>(BB_ORDER_MIN, BB_ORDER_MIN * 3 / 4 * (nb + 2) / nb);
  if (const char* e = std::getenv("MSC_B200_BB_ORDER")) {
    least = std::atoll(e);
    if (least < 0) least = INT64_MAX;
  }
  P.words = prune_mask_words(std::max<int64_t>(P.max_nb, 1), 256);
  P.npg = round_up(n, 256);
  // candidate lists of a launch within 1 GB (and the batches its parameters hold)
  P.group = int(std::min<int64_t>(std::min(nb, BB_GROUP),
                                  std::max<int64_t>(1, (int64_t(1) << 28) /
                                                           std::max<int64_t>(1, n * P.kprime))));
  P.ordered = P.candidates && P.kprime <= 32 && P.cfg.bn == 256 && d <= MSC_MAX_D && n >= least &&
              n >= 1024;
  return P;
}

size_t bb_workspace_bytes(const BbPlan& P) {
  BbWs w;
  return bb_carve(P, nullptr, w);
}

size_t bb_carve(const BbPlan& P, void* base, BbWs& w) {
  Carver c(base);
  w.ctl = c.take<Ctl>(1);
  w.km = c.take<KeyMax>(1);
  w.seg = c.take<SegDesc>(1);
  w.nfail = c.take<int32_t>(1);
  w.counters = c.take<int32_t>(std::max(P.nb, 1));
  w.perm = c.take<int32_t>(P.npk);
  w.qmap = c.take<int32_t>(P.n);
  w.flag = c.take<int32_t>(P.n);
  w.S = c.take<int64_t>(P.n + 1);
  w.scan = c.take<int64_t>(scan_i32_scratch_elems(P.n));
  w.fail_rows = c.take<int32_t>(P.n);
  w.mean = c.take<double>(P.d);
  w.partial = c.take<double>(colmean_partial_elems(1, P.d, BB_COLMEAN_NB));
  if (P.candidates) {
    const size_t el = P.prec == PREC_FP16 ? sizeof(__half) : sizeof(__nv_bfloat16);
    w.Aop = c.take<char>(size_t(round_up(P.n, QTILE)) * P.L.kp * el);
    w.Bop = c.take<char>(size_t(P.p1) * P.L.kp * el);
    w.qs = c.take<QStat>(P.npk);
    const int lists = P.ordered ? P.group : 1;
    w.items = c.take<WorkItem>(std::max<int64_t>(P.ntiles * lists, 1));
    w.cand_idx = c.take<int32_t>(size_t(P.n) * P.kprime * lists);
    w.cand_thr = c.take<float>(size_t(P.n) * lists);
    if (P.ordered) {
      w.gperm = c.take<int32_t>(P.npg);
      w.order_bytes = order_workspace_bytes(P.npg, P.d, BB_ORDER_LEAF);
      w.order_ws = c.take<char>(w.order_bytes);
      w.pitems = c.take<WorkItem>(P.ntiles * lists);
      w.pr = carve_query_prune(c, P.n, P.npk, P.p1, P.d, lists, P.ntiles * lists, P.words);
      w.fail_rows = c.take<int32_t>(size_t(P.n) * lists);
      w.fail_bat = c.take<int32_t>(size_t(P.n) * lists);
    }
  } else {
    w.Aop = w.Bop = nullptr;
    w.qs = nullptr;
    w.items = nullptr;
    w.cand_idx = nullptr;
    w.cand_thr = nullptr;
  }
  return c.bytes();
}

namespace {
// one centring and one scale, the operands of both sides (perm, qmap in place)
int bb_operands(const BbPlan& P, const BbWs& w, const float* X, cudaStream_t st) {
  MSC_TRY(launch_single_segment(w.seg, P.n, st));
  MSC_TRY(launch_colmean(X, w.seg, 1, P.n, P.d, w.partial, BB_COLMEAN_NB, w.mean,
                         &w.ctl->stats[MSC_STAT_NONFINITE], st));
  if (P.prec == PREC_FP16) MSC_TRY(launch_maxnorm(X, w.seg, 1, w.mean, P.d, P.n, w.ctl, st));
  MSC_TRY(launch_pack_tc(P.prec, X, w.perm, w.seg, 1, w.mean, P.d, P.p1, nullptr, nullptr, 0,
                         nullptr, w.Bop, w.qs, w.km, w.ctl, st));
  // the query operand: every cell, listed through qmap (the listed-row count in ctl)
  bb_set_i32_kernel<<<1, 1, 0, st>>>(&w.ctl->n_refine, int32_t(P.n));
  MSC_LAUNCH_CHECK();
  const size_t row = size_t(P.L.kp) * (P.prec == PREC_FP16 ? sizeof(__half) : sizeof(__nv_bfloat16));
  const int64_t tail = round_up(P.n, QTILE) - P.n;        // the operand's rows past the last query
  if (tail > 0)
    MSC_CUDA_TRY(cudaMemsetAsync(static_cast<char*>(w.Aop) + size_t(P.n) * row, 0, tail * row, st));
  return launch_pack_tc(P.prec, X, w.perm, w.seg, 1, w.mean, P.d, P.npk, w.qmap,
                        &w.ctl->n_refine, P.n, w.Aop, nullptr, w.qs, nullptr, w.ctl, st);
}

int run_bbknn_ordered(const BbPlan& P, const BbWs& w, const float* X, const int32_t* codes,
                      const int64_t* counts, int32_t* knn_idx, float* knn_dist,
                      cudaStream_t st) {
  const int g = grid_for(P.n, BB_T);
  // all cells in locality order, cells of no dense region last
  MSC_TRY(launch_single_segment(w.seg, P.n, st));
  int levels = 4;
  while ((int64_t(BB_ORDER_LEAF) << (levels - 4)) < P.n) ++levels;
  MSC_TRY(launch_order(X, P.d, w.seg, 1, P.npg, levels, BB_ORDER_LEAF, w.gperm, w.pr.leaf,
                       w.order_ws, w.order_bytes, st, P.n));
  MSC_TRY(launch_order_outliers(X, P.d, w.seg, P.n, P.npg, w.gperm, w.pr.leaf, w.pr, st));
  // layout: every batch's keys in that order, then the queries
  int32_t* leaf = w.pr.leaf2;                             // by packed row
  MSC_CUDA_TRY(cudaMemsetAsync(leaf, 0xFF, sizeof(int32_t) * P.npk, st));
  int64_t poff = 0;
  for (int b = 0; b < P.nb; ++b) {
    bb_flag_order_kernel<<<g, BB_T, 0, st>>>(codes, w.gperm, P.n, b, w.flag);
    MSC_LAUNCH_CHECK();
    MSC_TRY(scan_excl_i32(w.flag, P.n, w.S, w.scan, st));
    bb_place_order_kernel<<<g, BB_T, 0, st>>>(w.flag, w.gperm, w.pr.leaf, P.n, w.S, poff,
                                              counts[b], w.perm, leaf);
    MSC_LAUNCH_CHECK();
    poff += round_up(std::max<int64_t>(counts[b], 1), SEG_PAD);
  }
  bb_query_order_kernel<<<g, BB_T, 0, st>>>(w.gperm, w.pr.leaf, P.n, P.p1, w.perm, leaf, w.qmap);
  MSC_LAUNCH_CHECK();
  MSC_TRY(bb_operands(P, w, X, st));
  MSC_CUDA_TRY(cudaMemsetAsync(w.pr.rpos, 0, sizeof(double) * P.npk, st));
  MSC_TRY(launch_query_balls(X, P.d, P.npk, P.p1, P.ntiles, w.perm, leaf, w.pr.rpos, w.pr, st));
  const int64_t arows = round_up(P.n, QTILE);
  const int gw = grid_for(P.n, BB_WARPS);
  poff = 0;
  int col0 = 0, b = 0;
  while (b < P.nb) {
    BbBatches B{};
    int m = 0;
    for (; b < P.nb && m < P.group; ++b) {
      const int kk = int(std::min<int64_t>(P.kwb, counts[b]));
      if (kk > 0) {
        B.poff[m] = int32_t(poff);
        B.nb[m] = int32_t(counts[b]);
        B.kk[m] = kk;
        B.col0[m] = col0;
        B.start[m] = m ? B.start[m - 1] + B.nb[m - 1] : 0;
        ++m;
      }
      col0 += kk;
      poff += round_up(std::max<int64_t>(counts[b], 1), SEG_PAD);
    }
    if (m == 0) continue;
    const int64_t n_items = P.ntiles * m;
    bb_group_items_kernel<<<grid_for(n_items, BB_T), BB_T, 0, st>>>(B, m, P.n, P.p1, w.items,
                                                                   w.pitems);
    MSC_LAUNCH_CHECK();
    // near pass, radii, plan, main scan
    MSC_TRY(launch_nearest_tiles(w.pitems, n_items, P.d, w.pr, P.words, st));
    auto scan = [&](bool main_scan) {
      int32_t* counter = &w.ctl->tc_counter[main_scan ? 0 : 2];
      MSC_CUDA_TRY(cudaMemsetAsync(counter, 0, sizeof(int32_t), st));
      return launch_knn_tc(P.prec, P.cfg, w.Aop, w.Bop, arows, P.p1, P.L.kp, P.L.kmma, w.items,
                           n_items, w.perm, w.qmap, nullptr, counter, w.ctl, P.kprime, w.cand_idx,
                           w.cand_thr, P.kprime * m, st, w.pr.mask, P.words, false, false,
                           main_scan ? w.pr.seed : nullptr, nullptr, nullptr, nullptr,
                           main_scan ? w.pr.claim : nullptr, 1, P.n);
    };
    MSC_TRY(scan(false));
    MSC_TRY(launch_query_plan(P.d, w.perm, P.p1, P.n, m, w.pitems, n_items, w.cand_thr, w.qs,
                              w.km, w.ctl, P.prec, P.L.kmma, w.pr, P.words, st));
    MSC_TRY(launch_claim_order(n_items, P.words, w.pr, st));
    MSC_TRY(scan(true));
    MSC_CUDA_TRY(cudaMemsetAsync(w.nfail, 0, sizeof(int32_t), st));
    bb_group_rerank_kernel<<<gw, BB_T, 0, st>>>(X, P.d, P.n, P.p1, w.perm, B, m, w.cand_idx,
                                                w.cand_thr, P.kprime, w.qs, w.km, w.ctl, P.prec,
                                                P.L.kmma, P.K, knn_idx, knn_dist, w.fail_rows,
                                                w.fail_bat, w.nfail,
                                                &w.ctl->stats[MSC_STAT_CERTIFIED]);
    MSC_LAUNCH_CHECK();
    // (the flags of the layout are done with: their buffer takes the list; the counters are zero
    // before the first group)
    if (b > m) MSC_CUDA_TRY(cudaMemsetAsync(w.counters, 0, sizeof(int32_t) * P.nb, st));
    bb_store_order_kernel<<<g, BB_T, 0, st>>>(codes, P.n, B, m, b - m, w.nfail, w.counters, w.flag);
    MSC_LAUNCH_CHECK();
    bb_group_scan_kernel<<<gw, BB_T, 0, st>>>(X, P.d, w.flag, B, w.fail_rows, w.fail_bat, w.nfail,
                                              P.K, knn_idx, knn_dist,
                                              &w.ctl->stats[MSC_STAT_RESCANNED]);
    MSC_LAUNCH_CHECK();
  }
  bb_merge_kernel<<<gw, BB_T, 0, st>>>(P.n, P.K, knn_idx, knn_dist);
  MSC_LAUNCH_CHECK();
  return MSC_OK;
}
}  // namespace

int run_bbknn(const BbPlan& P, const BbWs& w, const float* X, const int32_t* codes,
              const int64_t* counts, int32_t* knn_idx, float* knn_dist, cudaStream_t st) {
  MSC_CUDA_TRY(cudaMemsetAsync(w.ctl, 0, sizeof(Ctl), st));
  MSC_CUDA_TRY(cudaMemsetAsync(w.km, 0, sizeof(KeyMax), st));
  MSC_CUDA_TRY(cudaMemsetAsync(w.counters, 0, sizeof(int32_t) * std::max(P.nb, 1), st));
  MSC_CUDA_TRY(cudaMemsetAsync(w.perm, 0xFF, sizeof(int32_t) * P.npk, st));
  const int g = grid_for(P.n, BB_T);
  if (P.ordered) return run_bbknn_ordered(P, w, X, codes, counts, knn_idx, knn_dist, st);
  // layout: batch segments, then the query region
  int64_t poff = 0;
  for (int b = 0; b < P.nb; ++b) {
    bb_flag_kernel<<<g, BB_T, 0, st>>>(codes, P.n, b, w.flag);
    MSC_LAUNCH_CHECK();
    MSC_TRY(scan_excl_i32(w.flag, P.n, w.S, w.scan, st));
    bb_place_kernel<<<g, BB_T, 0, st>>>(codes, P.n, b, w.S, poff, counts[b], w.perm);
    MSC_LAUNCH_CHECK();
    poff += round_up(std::max<int64_t>(counts[b], 1), SEG_PAD);
  }
  bb_query_region_kernel<<<g, BB_T, 0, st>>>(P.n, P.p1, w.perm, w.qmap);
  MSC_LAUNCH_CHECK();
  const int gw = grid_for(P.n, BB_WARPS);                 // one warp per cell
  if (P.candidates) {
    MSC_TRY(bb_operands(P, w, X, st));
  }
  poff = 0;
  int col0 = 0;
  for (int b = 0; b < P.nb; ++b) {
    const int64_t nbk = counts[b];
    const int kk = int(std::min<int64_t>(P.kwb, nbk));
    if (kk > 0) {
      if (P.candidates) {
        bb_items_kernel<<<grid_for(P.ntiles, BB_T), BB_T, 0, st>>>(P.n, poff, nbk, w.items);
        MSC_LAUNCH_CHECK();
        // the query operand's map spans its zero-filled tail rows too (no box beyond the rows)
        MSC_TRY(launch_knn_tc(P.prec, P.cfg, w.Aop, w.Bop, round_up(P.n, QTILE), P.p1, P.L.kp,
                              P.L.kmma, w.items, P.ntiles, w.perm, w.qmap, nullptr,
                              &w.counters[b], w.ctl,
                              P.kprime, w.cand_idx, w.cand_thr, P.kprime, st));
        MSC_CUDA_TRY(cudaMemsetAsync(w.nfail, 0, sizeof(int32_t), st));
        bb_rerank_kernel<<<gw, BB_T, 0, st>>>(X, P.d, P.n, P.p1, w.cand_idx, w.cand_thr,
                                              P.kprime, w.qs, w.km, w.ctl, P.prec, P.L.kmma, nbk,
                                              kk, P.K, col0, knn_idx, knn_dist, w.fail_rows,
                                              w.nfail, &w.ctl->stats[MSC_STAT_CERTIFIED]);
        MSC_LAUNCH_CHECK();
        bb_scan_kernel<<<gw, BB_T, 0, st>>>(X, P.d, P.n, w.perm, poff, nbk, w.fail_rows,
                                            w.nfail, kk, P.K, col0, knn_idx, knn_dist,
                                            &w.ctl->stats[MSC_STAT_RESCANNED]);
        MSC_LAUNCH_CHECK();
      } else {
        bb_scan_kernel<<<gw, BB_T, 0, st>>>(X, P.d, P.n, w.perm, poff, nbk, nullptr, nullptr,
                                            kk, P.K, col0, knn_idx, knn_dist,
                                            &w.ctl->stats[MSC_STAT_RESCANNED]);
        MSC_LAUNCH_CHECK();
      }
    }
    col0 += kk;
    poff += round_up(std::max<int64_t>(nbk, 1), SEG_PAD);
  }
  bb_merge_kernel<<<gw, BB_T, 0, st>>>(P.n, P.K, knn_idx, knn_dist);
  MSC_LAUNCH_CHECK();
  return MSC_OK;
}

size_t bb_distances_workspace_bytes(int64_t n) {
  Carver c(nullptr);
  c.take<int32_t>(n);
  c.take<int64_t>(scan_i32_scratch_elems(n));
  return c.bytes();
}

int launch_bb_distances(const int32_t* idx, const float* dist, int64_t n, int K, int64_t* indptr,
                        int32_t* indices, float* data, void* ws, cudaStream_t st) {
  Carver c(ws);
  int32_t* cnt = c.take<int32_t>(n);
  int64_t* scan = c.take<int64_t>(scan_i32_scratch_elems(n));
  bb_dist_count_kernel<<<grid_for(n, BB_T), BB_T, 0, st>>>(idx, dist, n, K, cnt);
  MSC_LAUNCH_CHECK();
  MSC_TRY(scan_excl_i32(cnt, n, indptr, scan, st));
  bb_dist_fill_kernel<<<grid_for(n, BB_WARPS), BB_T, 0, st>>>(idx, dist, n, K, indptr, indices,
                                                              data);
  MSC_LAUNCH_CHECK();
  return MSC_OK;
}

size_t trim_workspace_bytes(int64_t n) {
  Carver c(nullptr);
  c.take<float>(n);
  c.take<int32_t>(n);
  c.take<int64_t>(scan_i32_scratch_elems(n));
  return c.bytes();
}

int launch_trim(const int64_t* indptr, const int32_t* indices, const float* data, int64_t n,
                int trim, int64_t* out_ptr, int32_t* out_idx, float* out_data, void* ws,
                cudaStream_t st) {
  Carver c(ws);
  float* theta = c.take<float>(n);
  int32_t* cnt = c.take<int32_t>(n);
  int64_t* scan = c.take<int64_t>(scan_i32_scratch_elems(n));
  trim_theta_kernel<<<grid_for(n, BB_WARPS), BB_T, 0, st>>>(indptr, data, n, trim, theta);
  MSC_LAUNCH_CHECK();
  trim_count_kernel<<<grid_for(n, BB_WARPS), BB_T, 0, st>>>(indptr, indices, data, n, theta, cnt);
  MSC_LAUNCH_CHECK();
  MSC_TRY(scan_excl_i32(cnt, n, out_ptr, scan, st));
  trim_fill_kernel<<<grid_for(n, BB_WARPS), BB_T, 0, st>>>(indptr, indices, data, n, theta,
                                                           out_ptr, out_idx, out_data);
  MSC_LAUNCH_CHECK();
  return MSC_OK;
}

}  // namespace msc
