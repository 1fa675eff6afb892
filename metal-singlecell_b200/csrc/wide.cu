// Exact kNN of every row by direct differences, for lists wider than the candidate kernels keep
// (k - 1 > 64: the neighbour search of doublet detection asks for 82 of 9,000 cells).
//
// Reference counterpart: the `_knn` call of scrublet (metalsinglecell preprocess.py:280-306, the
// search itself neighbors.py:82-132).  Ranking every key in FP64 with a sorted list per row costs
// an FP64 difference per dimension and key and a merge of sorted lists for most batches of 32
// keys.  Here FP32 differences decide all but the keys around the k-th place:
//
//   1. sample   FP32 squared distances to m keys spread evenly over the sample's positions (all
//               keys when m reaches them); a bisection over their bit patterns takes a value T of
//               sample rank r, so that about 4 times k - 1 of all keys lie at or below it;
//   2. collect  FP32 distances to every key; those at or below T' = T·(1 + 8δ) are appended to the
//               row's buffer (δ = (d+4)·2^-24, the FP32 sum's relative error bound);
//   3. select   B = the (k-1)-th smallest FP32 value of the buffer; the keys within B·(1 + 3δ) + 2φ
//               are recomputed in FP64 (dimension order) and ordered by (FP64 value, index).
//               φ (F32_SQ_FLOOR) covers the roundings of sums below FP32's normal range.
//
// A key left out in step 2 has an FP32 value above T', hence a squared distance above (T'-φ)/(1+δ);
// the row is exact when its (k-1)-th FP64 value is below that, else (too few or too many collected,
// non-finite values) it is listed for the FP64 scan.  Which T the sample gives decides only how
// many keys are collected, never the result.
//
// Step 2 is the work: 2 FP32 instructions per dimension and pair.  A block takes 32 rows (4 per
// warp) against tiles of 128 keys: a lane holds 4 keys x 4 rows of sums, so that per dimension 4
// key reads and one 16-byte read of the rows serve 16 pairs, and a staged key serves 32 rows (with 8
// rows a block the element-wise copies into padded rows bounded it).  The next tile is copied while
// the current one is worked on, and the keys are split over blocks until the SMs are full.
// 9,000 x 30, k = 82: 0.66 ms; the FP64 scan of every key 3.75 ms, one kernel for the three
// steps with 8 rows a block 2.23 (plain staging), 0.97 (asynchronous copies).
#include "kernels.cuh"
#include "msc_warpsort.cuh"

namespace msc {

namespace {

__device__ unsigned long long g_wide_rows;      // rows finished, while profiling

constexpr int WD_CAP_PER_SLOT = 8;        // buffer entries per list entry
constexpr int WD_SAMPLE_MIN = 512, WD_SAMPLE_MAX = 4096;
constexpr size_t WD_SMEM_MAX = size_t(227) * 1024 - 1024;
constexpr int64_t WD_BUF_BYTES = int64_t(64) << 20;     // buffers of the rows in flight

int wide_slots(int kk) { return kk <= 128 ? 4 : (kk <= 256 ? 8 : 16); }
int wide_cap(int kk) { return 32 * wide_slots(kk) * WD_CAP_PER_SLOT; }
// rows whose buffers are in flight at once (a multiple of 256)
int64_t wide_rows(int64_t npacked, int kk) {
  return min64(npacked, WD_BUF_BYTES / (int64_t(wide_cap(kk)) * sizeof(int2)) / 256 * 256);
}

// keys sampled of n for lists of kk: x >= 6 of the kk nearest keys are expected among them
__host__ __device__ inline int wide_sample(int64_t n, int kk) {
  if (n <= WD_SAMPLE_MIN) return int(n);
  const int64_t want = (6 * n / kk + 127) / 128 * 128;
  return int(min64(n, max64(WD_SAMPLE_MIN, min64(want, WD_SAMPLE_MAX))));
}
// Sample rank of T: the expected rank x of the kk-th key and as far above it as a Poisson count of
// mean x goes once in some million rows (a row that exceeds it takes the FP64 scan, half a
// millisecond for one row).  Five standard deviations of that rank up still land below the buffer's
// 8 kk keys for x >= 6.
__device__ inline int wide_rank(int64_t n, int m, int kk) {
  if (m >= n) return kk;
  const float x = float(kk) * float(m) / float(n);
  return min(m, int(ceilf(x + 5.f * sqrtf(x))) + 4);
}

__device__ __forceinline__ void copy4_async(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ double wide_d2(const float* __restrict__ x, const float* __restrict__ y,
                                          int d) {
  double acc = 0.0;
#pragma unroll 4
  for (int t = 0; t < d; ++t) {
    const double df = double(x[t]) - double(y[t]);
    acc += df * df;
  }
  return acc;
}

// FP32 squared distances of KM staged keys (rows `ystride` apart, keys 32 lanes apart) to 4 rows
// (x: [d][NQ], 16-byte aligned)
template <int KM, int NQ>
__device__ __forceinline__ void tile_d2(const float* y, int ystride, const float* x, int d,
                                        float (&a)[KM][4]) {
#pragma unroll
  for (int v = 0; v < KM; ++v)
#pragma unroll
    for (int u = 0; u < 4; ++u) a[v][u] = 0.f;
#pragma unroll 2
  for (int t = 0; t < d; ++t) {
    const float4 q = *reinterpret_cast<const float4*>(x + t * NQ);
#pragma unroll
    for (int v = 0; v < KM; ++v) {
      const float w = y[v * 32 * ystride + t];
      const float e0 = q.x - w, e1 = q.y - w, e2 = q.z - w, e3 = q.w - w;
      a[v][0] = fmaf(e0, e0, a[v][0]);
      a[v][1] = fmaf(e1, e1, a[v][1]);
      a[v][2] = fmaf(e2, e2, a[v][2]);
      a[v][3] = fmaf(e3, e3, a[v][3]);
    }
  }
}

// ---- 1. sample: a block per 8 rows (two groups of 4, two warps of 64 keys each), a warp per row's
// threshold; padding rows get -1 (they collect nothing) ----
constexpr int SM_T = 128, SM_Q = 8, SM_KEYS = 128;
size_t sample_smem(int d, int m) {
  return sizeof(float) * (size_t(d) * SM_Q + size_t(2) * SM_KEYS * (d | 1) + size_t(SM_Q) * m);
}
__global__ void __launch_bounds__(SM_T)
wide_sample_kernel(const float* __restrict__ X, int d, const int32_t* __restrict__ perm,
                   const SegDesc* __restrict__ seg, int nseg, int64_t npacked, int m_max, int kk,
                   int cap, float* __restrict__ thr, int32_t* __restrict__ cnt) {
  extern __shared__ __align__(16) float wd_smem[];
  float* xq = wd_smem;                                  // [d][SM_Q]
  float* ys = xq + d * SM_Q;                            // two tiles [SM_KEYS][d | 1]
  const int ystride = d | 1, ytile = SM_KEYS * ystride;
  float* dist = ys + 2 * ytile;                         // [SM_Q][m]
  const int tid = threadIdx.x, lane = lane_id(), wib = warp_id();
  const int q0 = (wib & 1) * 4, key = (wib >> 1) * 64 + lane;         // keys key, key + 32
  const float delta = float(d + 4) * 0x1p-24f;
  for (int64_t p0 = int64_t(blockIdx.x) * SM_Q; p0 < npacked; p0 += int64_t(gridDim.x) * SM_Q) {
    // samples are padded to a multiple of 256 rows: the 8 rows belong to one
    const int sidx = find_seg(seg, nseg, p0);
    const int64_t off = seg[sidx].off, ns = seg[sidx].n;
    if (tid < SM_Q) cnt[p0 + tid] = 0;
    if (p0 - seg[sidx].poff >= ns) {                    // padding rows only (block-uniform)
      if (tid < SM_Q) thr[p0 + tid] = -1.f;
      continue;
    }
    const int m = min(m_max, wide_sample(ns, kk));
    __syncthreads();                                    // the previous rows' values are read
    for (int e = tid; e < d * SM_Q; e += SM_T) {
      const int q = e / d, t = e - q * d;
      const int32_t i = perm[p0 + q];
      xq[t * SM_Q + q] = i >= 0 ? X[int64_t(i) * d + t] : 0.f;
    }
    int self[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) self[u] = perm[p0 + q0 + u];
    // key e of the sample is the sample's cell floor(e·step / 2^32)
    const uint64_t step = (uint64_t(ns) << 32) / uint64_t(m);
    auto stage = [&](int base, float* tile) {
      for (int r = wib; r < SM_KEYS && base + r < m; r += SM_T / 32) {   // a warp per key
        const float* src = X + (off + int64_t((uint64_t(base + r) * step) >> 32)) * d;
        for (int t = lane; t < d; t += 32) copy4_async(tile + r * ystride + t, src + t);
      }
      copy_commit();
    };
    stage(0, ys);
    for (int base = 0, x = 0; base < m; base += SM_KEYS, x ^= 1) {
      copy_wait();
      __syncthreads();                                  // tile x is here, tile x ^ 1 is read
      if (base + SM_KEYS < m) stage(base + SM_KEYS, ys + (x ^ 1) * ytile);
      float a[2][4];
      tile_d2<2, SM_Q>(ys + x * ytile + key * ystride, ystride, xq + q0, d, a);
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        const int e = base + key + 32 * v;
        if (e >= m) continue;
        const int64_t j = off + int64_t((uint64_t(e) * step) >> 32);
#pragma unroll
        for (int u = 0; u < 4; ++u) dist[(q0 + u) * m + e] = j == self[u] ? F_INF : a[v][u];
      }
    }
    __syncthreads();
    for (int w = wib; w < SM_Q; w += SM_T / 32) {       // a warp per row: its threshold
      // non-negative floats order as their bits; NaN above all
      const float* v = dist + w * m;
      unsigned lo = 0xffffffffu, hi = 0u;
      for (int e = lane; e < m; e += 32) {
        const unsigned b = __float_as_uint(v[e]);
        lo = min(lo, b);
        hi = max(hi, b);
      }
      lo = __reduce_min_sync(FULL, lo);
      hi = __reduce_max_sync(FULL, hi);
      const int r = wide_rank(ns, m, kk), slack = max(2, r / 8);
      int below = m;                                    // values at or below hi
      // the smallest pattern with at least r values at or below it, or one with few more than r
      while (lo < hi) {
        const unsigned mid = lo + (hi - lo) / 2;
        int c = 0;
#pragma unroll 4
        for (int e = lane; e < m; e += 32) c += __float_as_uint(v[e]) <= mid;
        c = __reduce_add_sync(FULL, c);
        if (c < r) {
          lo = mid + 1;
        } else {
          hi = mid;
          below = c;
        }
        if (c >= r && c <= r + slack) break;
      }
      // A sample with many more values at or below it than r (coincident cells) says that more
      // keys than the buffer takes lie there: the row goes to the FP64 scan with nothing collected
      // (9,000 equal cells, k = 83, 5.03 -> 2.94 ms).
      const float T = __uint_as_float(hi) * (1.f + 8.f * delta);
      const bool fits = int64_t(below) * ns <= int64_t(cap) * m;
      if (lane == 0) thr[p0 + w] = fits && perm[p0 + w] >= 0 ? T : -1.f;
    }
  }
}

// ---- 2. collect: a block per 32 rows (4 per warp) and range of key tiles ----
constexpr int CO_T = 256, CO_Q = 32, CO_KM = 4, CO_KEYS = 32 * CO_KM;
size_t collect_smem(int d) {
  return sizeof(float) * (size_t(d) * CO_Q + size_t(2) * CO_KEYS * (d | 1));
}
__global__ void __launch_bounds__(CO_T, 4)
wide_collect_kernel(const float* __restrict__ X, int d, const int32_t* __restrict__ perm,
                    const SegDesc* __restrict__ seg, int nseg, int64_t row0, int64_t nrows,
                    const float* __restrict__ thr, int cap, int32_t* __restrict__ cnt,
                    int2* __restrict__ buf) {
  extern __shared__ __align__(16) float wd_smem[];
  float* xq = wd_smem;                                  // [d][CO_Q]
  float* ys = xq + d * CO_Q;                            // two tiles [CO_KEYS][d | 1]
  const int ystride = d | 1, ytile = CO_KEYS * ystride;
  const int tid = threadIdx.x, lane = lane_id(), wib = warp_id();
  const int q0 = wib * 4;
  const int64_t p0 = row0 + int64_t(blockIdx.x) * CO_Q;
  const int sidx = find_seg(seg, nseg, p0);
  const int64_t off = seg[sidx].off, ns = seg[sidx].n;
  if (p0 - seg[sidx].poff >= ns) return;                // padding rows only
  const int64_t tiles = (ns + CO_KEYS - 1) / CO_KEYS;
  const int64_t b0 = tiles * blockIdx.y / gridDim.y * CO_KEYS;
  const int64_t b1 = min64(ns, tiles * (blockIdx.y + 1) / gridDim.y * CO_KEYS);
  if (b0 >= b1) return;
  for (int e = tid; e < d * CO_Q; e += CO_T) {
    const int q = e / d, t = e - q * d;
    const int32_t i = perm[p0 + q];
    xq[t * CO_Q + q] = i >= 0 ? X[int64_t(i) * d + t] : 0.f;
  }
  int self[4];
  float T[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    self[u] = perm[p0 + q0 + u];
    T[u] = thr[p0 + q0 + u];                            // -1 for padding rows
  }
  // a tile's rows are one run of memory, copied element by element into padded rows
  const int dr = CO_T / d, dt = CO_T - dr * d;          // a step of CO_T elements: rows, dimensions
  const int r_first = tid / d, t_first = tid - r_first * d;
  auto stage = [&](int64_t base, float* tile) {
    const int ne = int(min64(CO_KEYS, b1 - base)) * d;
    const float* src = X + (off + base) * d;
    int r = r_first, t = t_first;
    for (int e = tid; e < ne; e += CO_T) {
      copy4_async(tile + r * ystride + t, src + e);
      r += dr;
      t += dt;
      if (t >= d) { t -= d; ++r; }
    }
    copy_commit();
  };
  stage(b0, ys);
  int x = 0;
  for (int64_t base = b0; base < b1; base += CO_KEYS, x ^= 1) {
    const int nk = int(min64(CO_KEYS, b1 - base));
    copy_wait();
    __syncthreads();                                    // tile x is here, tile x ^ 1 is read
    if (base + CO_KEYS < b1) stage(base + CO_KEYS, ys + (x ^ 1) * ytile);
    float a[CO_KM][4];
    tile_d2<CO_KM, CO_Q>(ys + x * ytile + lane * ystride, ystride, xq + q0, d, a);
#pragma unroll
    for (int v = 0; v < CO_KM; ++v) {
      const int r = lane + 32 * v;
      if (r >= nk) continue;
      const int j = int(off + base) + r;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (a[v][u] <= T[u] && j != self[u]) {
          const int at = atomicAdd(&cnt[p0 + q0 + u], 1);
          if (at < cap)
            buf[(p0 - row0 + q0 + u) * cap + at] = make_int2(__float_as_int(a[v][u]), j);
        }
    }
  }
}

// ---- 3. select: a warp per row ----
constexpr int SE_WARPS = 4;
template <int SLOTS>
__global__ void __launch_bounds__(SE_WARPS * 32)
wide_select_kernel(const float* __restrict__ X, int d, const int32_t* __restrict__ perm,
                   int64_t row0, int64_t nrows, const float* __restrict__ thr,
                   const int32_t* __restrict__ cnt, const int2* __restrict__ buf, int cap, int k,
                   int cosine, int32_t* __restrict__ knn_idx, float* __restrict__ knn_dist,
                   int32_t* __restrict__ fail_rows, Ctl* __restrict__ ctl, int prof) {
  __shared__ int win_all[SE_WARPS][32 * SLOTS];
  __shared__ double val_all[SE_WARPS][32 * SLOTS];
  __shared__ __align__(16) float xs_all[SE_WARPS][MSC_MAX_D];
  const int lane = lane_id(), wib = warp_id(), kk = k - 1;
  int* win = win_all[wib];
  double* val = val_all[wib];
  float* xs = xs_all[wib];
  const float delta = float(d + 4) * 0x1p-24f;
  const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  int done = 0;
  for (int64_t rr = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5; rr < nrows;
       rr += nwarps) {
    const int64_t p = row0 + rr;
    const int32_t i = perm[p];
    if (i < 0) continue;                                // warp-uniform
    const int c = cnt[p];
    const int2* mine = buf + rr * cap;
    bool ok = c >= kk && c <= cap;
    if (ok) {
      __syncwarp();                                     // the previous row's values are read
      for (int t = lane; t < d; t += 32) xs[t] = X[int64_t(i) * d + t];
      unsigned lo = 0u, hi = __float_as_uint(thr[p]);
      while (lo < hi) {                                 // the kk-th smallest bit pattern
        const unsigned mid = lo + (hi - lo) / 2;
        int n_le = 0;
#pragma unroll 4
        for (int e = lane; e < c; e += 32) n_le += unsigned(mine[e].x) <= mid;
        if (__reduce_add_sync(FULL, n_le) < kk) lo = mid + 1;
        else hi = mid;
      }
      const double lim = double(__uint_as_float(hi)) * (1.0 + 3.0 * double(delta)) + 2.0 * F32_SQ_FLOOR;
      int w = 0;                                        // the window's keys
      for (int e0 = 0; e0 < c; e0 += 32) {
        const int e = e0 + lane;
        const int2 x = e < c ? mine[e] : make_int2(0x7f800000, 0);
        const bool in = e < c && double(__int_as_float(x.x)) <= lim;
        const unsigned b = __ballot_sync(FULL, in);
        const int at = w + __popc(b & ((1u << lane) - 1u));
        if (in && at < 32 * SLOTS) win[at] = x.y;
        w += __popc(b);
      }
      __syncwarp();
      ok = w <= 32 * SLOTS;
      if (ok) {
        for (int e = lane; e < w; e += 32) val[e] = wide_d2(xs, X + int64_t(win[e]) * d, d);
        __syncwarp();
        // each entry's place is the number of entries before it in (value, index) order; the
        // window is a few more than kk entries, and counting is one broadcast read and SLOTS
        // comparisons each where a sorted list takes a network per 32 entries
        double g[SLOTS];
        int id[SLOTS], rank[SLOTS];
#pragma unroll
        for (int s = 0; s < SLOTS; ++s) {
          const int e = s * 32 + lane;
          g[s] = e < w ? val[e] : 0.0;
          id[s] = e < w ? win[e] : 0;
          rank[s] = 0;
        }
        for (int f = 0; f < w; ++f) {
          const double vf = val[f];
          const int jf = win[f];
#pragma unroll
          for (int s = 0; s < SLOTS; ++s)
            if (s * 32 < w) rank[s] += dless(vf, jf, g[s], id[s]);
        }
        bool below = false;                             // the kk-th value is below the bound
        const double bound = (double(thr[p]) - F32_SQ_FLOOR) / (1.0 + double(delta));
#pragma unroll
        for (int s = 0; s < SLOTS; ++s)
          below = below || (s * 32 + lane < w && rank[s] == kk - 1 && g[s] < bound);
        ok = __any_sync(FULL, below);
        if (ok) {
          if (lane == 0) { knn_idx[int64_t(i) * k] = i; knn_dist[int64_t(i) * k] = 0.f; ++done; }
#pragma unroll
          for (int s = 0; s < SLOTS; ++s)
            if (s * 32 + lane < w && rank[s] < kk) {
              knn_idx[int64_t(i) * k + 1 + rank[s]] = id[s];
              knn_dist[int64_t(i) * k + 1 + rank[s]] =
                  cosine ? __double2float_rn(g[s] * 0.5) : __double2float_rn(sqrt(g[s]));
            }
        }
      }
    }
    if (!ok && lane == 0) {
      fail_rows[atomicAdd(&ctl->n_fail, 1)] = int32_t(p);
    }
  }
  if (lane == 0 && done)
    atomicAdd(reinterpret_cast<unsigned long long*>(&ctl->stats[MSC_STAT_RESCANNED]),
              (unsigned long long)done);
  if (prof && lane == 0 && done) atomicAdd(&g_wide_rows, (unsigned long long)done);
}

}  // namespace

bool wide_scan_ok(int64_t max_seg, int d, int k) {
  const int kk = k - 1, m = wide_sample(max_seg, kk);
  if (kk < 1 || kk > 512 || (m < max_seg && double(kk) * m < 5.9 * double(max_seg))) return false;
  return sample_smem(d, m) <= WD_SMEM_MAX && collect_smem(d) <= WD_SMEM_MAX;
}

int wide_counter(unsigned long long* out) {
  MSC_CUDA_TRY(cudaMemcpyFromSymbol(out, g_wide_rows, sizeof(*out)));
  return MSC_OK;
}
int wide_counter_clear() {
  const unsigned long long z = 0;
  MSC_CUDA_TRY(cudaMemcpyToSymbol(g_wide_rows, &z, sizeof(z)));
  return MSC_OK;
}

WideWs carve_wide(Carver& c, int64_t npacked, int k) {
  WideWs w{};
  w.thr = c.take<float>(npacked);
  w.cnt = c.take<int32_t>(npacked);
  w.buf = c.take<int2>(size_t(wide_rows(npacked, k - 1)) * wide_cap(k - 1));
  return w;
}

int launch_wide_scan(const float* X, int d, const int32_t* perm, const SegDesc* seg, int nseg,
                     int64_t npacked, int64_t max_seg, int k, int cosine, const WideWs& ws,
                     int32_t* knn_idx, float* knn_dist, int32_t* fail_rows, Ctl* ctl,
                     cudaStream_t st) {
  const int kk = k - 1, cap = wide_cap(kk), sms = num_sms();
  const int m = wide_sample(max_seg, kk);               // at least every smaller sample's
  const size_t ssm = sample_smem(d, m), csm = collect_smem(d);
  MSC_CUDA_TRY(raise_smem_cap(wide_sample_kernel, ssm));
  MSC_CUDA_TRY(raise_smem_cap(wide_collect_kernel, csm));
  const int sgrid = int(std::min<int64_t>(npacked / SM_Q, int64_t(sms) * 64));
  wide_sample_kernel<<<sgrid, SM_T, ssm, st>>>(X, d, perm, seg, nseg, npacked, m, kk, cap,
                                               ws.thr, ws.cnt);
  MSC_LAUNCH_CHECK();
  const int64_t rows = wide_rows(npacked, kk);
  const int prof = profiling_enabled() ? 1 : 0;
  const int resident = sms * resident_blocks_fn(reinterpret_cast<const void*>(wide_collect_kernel),
                                                CO_T, csm);
  for (int64_t r0 = 0; r0 < npacked; r0 += rows) {
    const int64_t nr = std::min(rows, npacked - r0);
    const int64_t bx = nr / CO_Q;
    // four waves' worth of blocks where the keys can be split that far (at least two tiles a block)
    const int64_t by = std::max<int64_t>(1, std::min<int64_t>(ceil_div(4 * resident, bx),
                                                              max_seg / (2 * CO_KEYS)));
    wide_collect_kernel<<<dim3(unsigned(bx), unsigned(by)), CO_T, csm, st>>>(
        X, d, perm, seg, nseg, r0, nr, ws.thr, cap, ws.cnt, ws.buf);
    MSC_LAUNCH_CHECK();
    const int g = int(std::max<int64_t>(1, std::min<int64_t>(ceil_div(nr, SE_WARPS),
                                                            int64_t(sms) * 64)));
    if (kk <= 128)
      wide_select_kernel<4><<<g, SE_WARPS * 32, 0, st>>>(X, d, perm, r0, nr, ws.thr, ws.cnt,
                                                         ws.buf, cap, k, cosine, knn_idx,
                                                         knn_dist, fail_rows, ctl, prof);
    else if (kk <= 256)
      wide_select_kernel<8><<<g, SE_WARPS * 32, 0, st>>>(X, d, perm, r0, nr, ws.thr, ws.cnt,
                                                         ws.buf, cap, k, cosine, knn_idx,
                                                         knn_dist, fail_rows, ctl, prof);
    else
      wide_select_kernel<16><<<g, SE_WARPS * 32, 0, st>>>(X, d, perm, r0, nr, ws.thr, ws.cnt,
                                                          ws.buf, cap, k, cosine, knn_idx,
                                                          knn_dist, fail_rows, ctl, prof);
    MSC_LAUNCH_CHECK();
  }
  return MSC_OK;
}

}  // namespace msc
