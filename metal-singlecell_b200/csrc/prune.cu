// Key-tile pruning for the tensor-core candidate kernel: the pairs of (query tile, key tile) that
// cannot contribute a candidate are never computed.
//
// The reference computes every distance of a row block (neighbors.py:114-119); so does the plain
// form here.  An exact kNN does not need to: a key whose squared distance to row x is provably
// above x's running k'-th value can never enter x's candidate list.  This file proves it per tile
// pair with bounding balls:
//
//   1. near pass: the candidate kernel visits only each query tile's own key tile (the cells are
//      in locality order) and returns every row's k'-th smallest value thr_x.
//      R_x = thr_x + |z_x|² + 3·eps_x bounds, in the scaled space z of the operands, the squared
//      distance below which x can still take a key (eps_x = the certificate's bound on the
//      operand and accumulation error, see rerank.cu);
//   2. outliers: rows whose R_x is far above their sample's mean R (cells in no dense region)
//      move to the end of their sample, so that the balls of the tiles of regular rows stay
//      tight; the order is otherwise kept (stable partition), and so are the locality-tree leaves;
//   3. balls: every 32-row block of packed rows gets two balls (split at the first leaf boundary
//      inside the block), every 128-row query tile and every 256-row block one ball; centres are
//      float, radii are rounded up so that each ball holds all of its rows;
//   4. plan: key tile K is skipped for query tile Q when every ball u of Q and every ball w of K
//      are separated: |c_u − c_w| − r_u − r_w = L > 0 and f²·L² > max R over u's rows.  Then every
//      (x, y) with x in Q, y in K has v(x,y) = |z_x − z_y|² − |z_x|² > thr_x + 3·eps_x, so the
//      approximate value the kernel would compute is above thr_x + 2·eps_x; the k' keys behind
//      thr_x are never skipped, so the final k'-th value T_x <= thr_x + 2·eps_x, and the
//      certificate's premise (every key outside the list has approximate value >= T_x) holds for
//      skipped keys exactly as for scanned ones.  Near tiles are always visited.
//
// Each query tile gets a bit mask over its sample's key tiles (set = visit, near tiles excluded);
// the candidate kernel walks its near tiles first and then the set bits in ascending order.
#include <cstdlib>

#include "kernels.cuh"

namespace msc {

namespace {

constexpr int PR_T = 256;

// summed over plans while profiling: key tiles visited beyond the near tiles, all such tiles,
// tiles that failed level 1, tiles that reached the pair tests, pair tests
__device__ unsigned long long g_prune_tiles[6];
constexpr int SUB = 32;          // rows per sub-block (two balls each)
constexpr float NO_BALL = -1.f;  // radius of a ball without rows
constexpr double OUTLIER_FACTOR = 4.0;   // default; MSC_B200_OUTLIER_FACTOR overrides (tuning)

__device__ __forceinline__ double warp_sum_d(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  return v;
}
__device__ __forceinline__ double warp_max_d(double v) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(FULL, v, o));
  return v;
}

// R per packed position of the near-pass layout (+inf where the row has no finite threshold;
// padding rows get NaN and are never read as rows)
__global__ void row_radius_kernel(const int32_t* __restrict__ perm, int64_t npacked,
                                  const float* __restrict__ cand_thr,
                                  const QStat* __restrict__ qs, const KeyMax* __restrict__ km,
                                  int prec, int kmma, int d, double* __restrict__ rpos) {
  for (int64_t p = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; p < npacked;
       p += int64_t(gridDim.x) * blockDim.x) {
    const int32_t i = perm[p];
    if (i < 0) { rpos[p] = __longlong_as_double(0x7ff8000000000000ll); continue; }
    const double thr = cand_thr[i];
    const QStat q = qs[p];
    const double r = thr + q.sq + 3.0 * cert_eps(q, *km, prec, kmma, d);
    rpos[p] = r < 1e300 ? r : __longlong_as_double(0x7ff0000000000000ll);
  }
}

// mean of the finite R of every sample, in two steps with a fixed summation order: MEAN_CHUNKS
// blocks per sample (grid y = sample) each sum a fixed slice, then one thread per sample adds the
// slices in order
constexpr int MEAN_CHUNKS = 64;
__global__ void sample_mean_partial_kernel(const SegDesc* __restrict__ seg, int nseg,
                                           const double* __restrict__ rpos,
                                           double2* __restrict__ part) {
  __shared__ double ssum[PR_T / 32], scnt[PR_T / 32];
  for (int sidx = blockIdx.y; sidx < nseg; sidx += gridDim.y) {
    const SegDesc s = seg[sidx];
    const int64_t per = (s.n + MEAN_CHUNKS - 1) / MEAN_CHUNKS;
    const int64_t j0 = int64_t(blockIdx.x) * per, j1 = min64(s.n, j0 + per);
    double sum = 0.0, cnt = 0.0;
    for (int64_t j = j0 + threadIdx.x; j < j1; j += blockDim.x) {
      const double r = rpos[s.poff + j];
      if (r < 1e300) { sum += r; cnt += 1.0; }
    }
    sum = warp_sum_d(sum);
    cnt = warp_sum_d(cnt);
    __syncthreads();
    if (lane_id() == 0) { ssum[warp_id()] = sum; scnt[warp_id()] = cnt; }
    __syncthreads();
    if (threadIdx.x == 0) {
      double a = 0.0, b = 0.0;
      for (int w = 0; w < int(blockDim.x >> 5); ++w) { a += ssum[w]; b += scnt[w]; }
      part[int64_t(sidx) * MEAN_CHUNKS + blockIdx.x] = make_double2(a, b);
    }
  }
}
__global__ void sample_mean_final_kernel(const double2* __restrict__ part, int nseg,
                                         double* __restrict__ mean_out) {
  for (int sidx = blockIdx.x * blockDim.x + threadIdx.x; sidx < nseg;
       sidx += gridDim.x * blockDim.x) {
    double a = 0.0, b = 0.0;
    for (int c = 0; c < MEAN_CHUNKS; ++c) {
      const double2 v = part[int64_t(sidx) * MEAN_CHUNKS + c];
      a += v.x;
      b += v.y;
    }
    mean_out[sidx] = b > 0.0 ? a / b : __longlong_as_double(0x7ff0000000000000ll);
  }
}

__global__ void regular_flag_kernel(const int32_t* __restrict__ perm, int64_t npacked,
                                    const SegDesc* __restrict__ seg, int nseg,
                                    const double* __restrict__ rpos,
                                    const double* __restrict__ mean, double factor,
                                    int32_t* __restrict__ reg) {
  for (int64_t p = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; p < npacked;
       p += int64_t(gridDim.x) * blockDim.x) {
    if (perm[p] < 0) { reg[p] = 0; continue; }
    const double m = mean[find_seg(seg, nseg, p)];
    reg[p] = rpos[p] > factor * m ? 0 : 1;                // NaN / inf mean: regular
  }
}

// stable partition inside every sample: regular rows first, then the outliers (leaf OUTLIER_LEAF)
// The seed of a row lies strictly above thr + 2·eps: the near pass's k' keys keep values at or
// below thr + 2·eps in the scan of the new layout (the operands of a row are the same; each value is within eps of
// the exact one), so the row's final k'-th value cannot exceed it.
__global__ void partition_kernel(const int32_t* __restrict__ perm, const int32_t* __restrict__ leaf,
                                 const double* __restrict__ rpos, int64_t npacked,
                                 const SegDesc* __restrict__ seg, int nseg,
                                 const int32_t* __restrict__ reg, const int64_t* __restrict__ S,
                                 const float* __restrict__ cand_thr, const QStat* __restrict__ qs,
                                 const KeyMax* __restrict__ km, int prec, int kmma, int d, int bn,
                                 int32_t* __restrict__ perm2, int32_t* __restrict__ leaf2,
                                 double* __restrict__ rpos2, float* __restrict__ seed2,
                                 int32_t* __restrict__ iperm, int4* __restrict__ excl) {
  for (int64_t p = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; p < npacked;
       p += int64_t(gridDim.x) * blockDim.x) {
    const SegDesc s = seg[find_seg(seg, nseg, p)];
    int64_t pos = p;
    int32_t lf = leaf[p];
    if (p < s.poff + s.n) {
      const int64_t before = S[p] - S[s.poff];                 // regular rows before p
      if (reg[p]) {
        pos = s.poff + before;
      } else {
        const int64_t nreg = S[s.poff + s.n] - S[s.poff];
        pos = s.poff + nreg + (p - s.poff) - before;
        lf = OUTLIER_LEAF;
      }
    }
    const int32_t i = perm[p];
    float sd = F_INF;
    if (i >= 0) {
      const double t = double(cand_thr[i]) + 2.0 * cert_eps(qs[p], *km, prec, kmma, d);
      if (t < 1e300) sd = nextafterf(__double2float_ru(t), F_INF);   // strictly above
    }
    perm2[pos] = i;
    leaf2[pos] = lf;
    rpos2[pos] = rpos[p];
    seed2[pos] = sd;
    int4 ex = make_int4(0, 0, 0, 0);
    if (i >= 0) {
      iperm[i] = int32_t(pos);
      // the near pass scored row i against key tile diag of its query tile (bn rows); those keys
      // are a run of regular rows and a run of outliers in the new order
      const int64_t qt = (p - s.poff) / QTILE;
      const int64_t a = s.poff + (qt * QTILE / bn) * bn, b = min64(a + bn, s.poff + s.n);
      const int64_t ra = S[a] - S[s.poff], rb = S[b] - S[s.poff];
      const int64_t nreg = S[s.poff + s.n] - S[s.poff];
      ex = make_int4(int(s.poff + ra), int(s.poff + rb), int(s.poff + nreg + (a - s.poff) - ra),
                     int(s.poff + nreg + (b - s.poff) - rb));
    }
    excl[pos] = ex;
  }
}

// Centres that lanes read for consecutive balls (key tiles, sub-balls) lie interleaved: balls in
// groups of 32, float4 t of ball g at [g / 32][t][g % 32], so that a warp's 32 reads of one float4 are
// 512 consecutive bytes.  (Row after row, 208 bytes apart at 50 dimensions, each read touched 32
// lines: the plan at 1.3M cells took 7.03 ms, 6.63 interleaved.)
__device__ __forceinline__ int64_t inter_at(int64_t g, int n4) {
  return (g >> 5) * (32 * n4) + (g & 31);
}
constexpr int INTER = 32;        // float4s from one to the next of an interleaved ball
__device__ __forceinline__ void store_centre(float* centre, int64_t g, int dp, int t, float v,
                                             bool interleaved) {
  if (interleaved)
    centre[(inter_at(g, dp / 4) + int64_t(t >> 2) * INTER) * 4 + (t & 3)] = v;
  else
    centre[g * dp + t] = v;
}

// Squared distance of a row to a centre (shared memory, float) by 8 lanes, FP64: every lane of the
// group returns it.  Four rows of a warp go at once, so a row's sum takes 3 shuffle steps for four
// rows where a warp a row takes 5 for one.
__device__ __forceinline__ double row_d2_8(const float* __restrict__ x, const float* c, int d,
                                           int sub) {
  double a = 0.0;
  for (int t = sub; t < d; t += 8) {
    const double u = double(x[t]) - double(c[t]);
    a += u * u;
  }
  a += __shfl_xor_sync(FULL, a, 4);
  a += __shfl_xor_sync(FULL, a, 2);
  a += __shfl_xor_sync(FULL, a, 1);
  return a;
}

// One ball per group of G packed rows (G = 128 or 256): centre = float(mean of the rows), radius =
// max distance to that centre, rounded up.  A block of eight warps per group, G / 8 rows each (one
// warp per group read 256 rows one after another, 157 us at any n up to 100,000).
template <int G, bool INTERLEAVED>
__global__ void __launch_bounds__(PR_T)
group_ball_kernel(const float* __restrict__ X, int d, int dp, const int32_t* __restrict__ perm,
                  int64_t ngroups, float* __restrict__ centre, float* __restrict__ radius) {
  constexpr int W = PR_T / 32, R = G / W;
  __shared__ double part[W][MSC_MAX_D];
  __shared__ float c[MSC_MAX_D];
  __shared__ double mxs[W];
  __shared__ int cnts[W];
  const int lane = lane_id(), wib = warp_id();
  for (int64_t g = blockIdx.x; g < ngroups; g += gridDim.x) {
    const int64_t p0 = g * G + wib * R;
    const int32_t my_i = lane < R ? perm[p0 + lane] : -1;
    double s[4] = {0, 0, 0, 0};
#pragma unroll 4
    for (int r = 0; r < R; ++r) {
      const int32_t i = __shfl_sync(FULL, my_i, r);
      if (i < 0) continue;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int t = lane + 32 * j;
        if (t < d) s[j] += X[int64_t(i) * d + t];
      }
    }
    __syncthreads();                           // the previous group's values are read
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (lane + 32 * j < d) part[wib][lane + 32 * j] = s[j];
    const unsigned have = __ballot_sync(FULL, my_i >= 0);
    if (lane == 0) cnts[wib] = __popc(have);
    __syncthreads();
    int cnt = 0;
    for (int w = 0; w < W; ++w) cnt += cnts[w];
    for (int t = threadIdx.x; t < dp; t += PR_T) {
      double a = 0.0;
      if (t < d)
        for (int w = 0; w < W; ++w) a += part[w][t];
      const float v = (cnt && t < d) ? float(a / cnt) : 0.f;
      c[t] = v;
      store_centre(centre, g, dp, t, v, INTERLEAVED);
    }
    __syncthreads();
    double mx = 0.0;
    for (int r = 0; r < R; r += 4) {
      const int32_t i = __shfl_sync(FULL, my_i, r + (lane >> 3));
      const double a = row_d2_8(X + int64_t(i < 0 ? 0 : i) * d, c, d, lane & 7);
      if (i >= 0) mx = fmax(mx, a);
    }
    mx = warp_max_d(mx);
    if (lane == 0) mxs[wib] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < W; ++w) mx = fmax(mx, mxs[w]);
      radius[g] = cnt ? __double2float_ru(sqrt(mx) * (1.0 + 0x1p-40)) : NO_BALL;
    }
  }
}

// Two balls per 32-row block, split at the first row whose leaf differs from the block's first
// row (rows of one leaf are close, rows of two leaves may lie in two clusters), and the block's
// max R.  Ball 2b covers rows [0, m), ball 2b+1 rows [m, 32).
__global__ void __launch_bounds__(PR_T)
sub_ball_kernel(const float* __restrict__ X, int d, int dp,
                                const int32_t* __restrict__ perm,
                                const int32_t* __restrict__ leaf,
                                const double* __restrict__ rpos, int64_t nsub,
                                float* __restrict__ centre, float* __restrict__ radius,
                                double* __restrict__ rsub) {
  __shared__ float c_all[PR_T / 32][MSC_MAX_D];
  const int lane = lane_id();
  float* c = c_all[warp_id()];
  const int64_t warps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t b = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5; b < nsub; b += warps) {
    const int64_t p0 = b * SUB;
    const int32_t my_i = perm[p0 + lane];
    const int32_t my_leaf = leaf[p0 + lane];
    const int32_t leaf0 = __shfl_sync(FULL, my_leaf, 0);
    const unsigned diff = __ballot_sync(FULL, my_leaf != leaf0);
    const int m = diff ? __ffs(diff) - 1 : SUB;
    // the block's max R over its rows (unknown radius = +inf)
    double rv = 0.0;
    if (my_i >= 0) {
      const double r = rpos[p0 + lane];
      rv = r < 1e300 ? r : __longlong_as_double(0x7ff0000000000000ll);
    }
    rv = warp_max_d(rv);
    if (lane == 0) rsub[b] = rv;
    for (int h = 0; h < 2; ++h) {
      const int r0 = h ? m : 0, r1 = h ? SUB : m;
      double s[4] = {0, 0, 0, 0};
      int cnt = 0;
#pragma unroll 4
      for (int r = r0; r < r1; ++r) {
        const int32_t i = __shfl_sync(FULL, my_i, r);
        if (i < 0) continue;
        ++cnt;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int t = lane + 32 * j;
          if (t < d) s[j] += X[int64_t(i) * d + t];
        }
      }
      __syncwarp();                              // the previous ball's centre is read
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int t = lane + 32 * j;
        const float v = (cnt && t < d) ? float(s[j] / cnt) : 0.f;
        if (t < dp) {
          c[t] = v;
          store_centre(centre, 2 * b + h, dp, t, v, true);
        }
      }
      __syncwarp();
      double mx = 0.0;
      for (int r = r0; r < r1; r += 4) {
        const int rr = r + (lane >> 3);
        const int32_t i = __shfl_sync(FULL, my_i, rr & 31);
        const bool in = rr < r1 && i >= 0;
        const double a = row_d2_8(X + int64_t(in ? i : 0) * d, c, d, lane & 7);
        if (in) mx = fmax(mx, a);
      }
      mx = warp_max_d(mx);
      if (lane == 0)
        radius[2 * b + h] = cnt ? __double2float_ru(sqrt(mx) * (1.0 + 0x1p-40)) : NO_BALL;
    }
  }
}

// Are the balls (cu, ru) and (cw, rw) so far apart that no row of u can take a key of w?  That is
// L = |cu - cw| - ru - rw > 0 and f²·L² > R·(1 + 1e-9) (R = max R over u's rows, z-space, f = the
// operand scale), which is |cu - cw| > ru + rw + reach with reach = sqrt(R·(1 + 1e-9)) / f: the root is
// taken once per ball u (ball_reach) and a test compares squares (its 1e-12 covers the FP64
// roundings).  An empty ball is separated from everything; an unknown R (reach +inf) from nothing.
// Centres are n4 float4 (zero padded), SA and SB float4s apart; the FP32 distance is lowered by its
// rounding bound (d+8 units of 2^-23 relative) before the test; what its square loses below FP32's
// normal range is in reach (far + a squared is at least far² + a²).
__device__ __forceinline__ double ball_reach(double R, double f) {
  return R < 1e300 ? sqrt(R * (1.0 + 1e-9)) / f + sqrt(F32_SQ_FLOOR)
                   : __longlong_as_double(0x7ff0000000000000ll);
}
template <int SA, int SB>
__device__ __forceinline__ float ball_d2(const float4* a, const float4* b, int n4) {
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll 4
  for (int t = 0; t < n4; ++t) {
    const float4 x = a[t * SA], y = b[t * SB];
    const float e0 = x.x - y.x, e1 = x.y - y.y, e2 = x.z - y.z, e3 = x.w - y.w;
    s0 = fmaf(e0, e0, s0);
    s1 = fmaf(e1, e1, s1);
    s2 = fmaf(e2, e2, s2);
    s3 = fmaf(e3, e3, s3);
  }
  return (s0 + s1) + (s2 + s3);
}
__device__ __forceinline__ bool apart(float d2, float ru, float rw, double reach, int d) {
  if (ru < 0.f || rw < 0.f) return true;
  const double lo = double(d2) * (1.0 - double(d + 8) * 0x1p-23);
  const double far = (double(ru) + double(rw) + reach) * (1.0 + 1e-12);
  return lo > far * far;
}
template <int SA, int SB>
__device__ __forceinline__ bool separated(const float4* a, float ru, double reach, const float4* b,
                                          float rw, int n4, int d) {
  return apart(ball_d2<SA, SB>(a, b, n4), ru, rw, reach, d);
}

// One warp per query tile (work item).  Level 1, lane = key tile: the query tile's ball against
// the 256-row ball holding the key tile.  The key tiles of a 32-tile chunk that fail it go to
// level 2 together: (a) every query sub-ball against the key tile's ball, (b) every key sub-ball
// against the query tile's ball — a sub-ball separated there is separated from every sub-ball of
// the other side — with the (key tile, sub-ball) tests spread over the lanes; then, per key tile
// left, the remaining sub-ball pairs, one pair per lane.
constexpr int PLAN_WARPS = 4;
// mask words (32 key tiles each) per warp task: at most 4, fewer while the tasks do not give every
// resident warp PLAN_TASKS of them.  The work of a task varies from one test a tile to some fifty, and
// at 100,000 cells the launch waited for the few warps with the most (0.73 ms with 8 words, 0.85 ms
// with the n-th set bits found by __fns, 0.12 ms now; 1.3M cells 6.63 -> 5.90 without __fns, 5.27
// with squared tests and 4-word tasks, 4.36 with the visits of level 1).
constexpr int PLAN_WORDS_MAX = 4, PLAN_TASKS = 16;
constexpr int PLAN_MAX_PAIRS = 32;  // sub-ball pairs tested per key tile (one per lane);
                                    // MSC_B200_PLAN_PAIRS overrides (tuning)
__global__ void __launch_bounds__(PLAN_WARPS * 32, 6)
plan_kernel(const WorkItem* __restrict__ items, int64_t n_items, int bn, int d, int dp,
            const Ctl* ctl, int prec, const float* __restrict__ qc, const float* __restrict__ qr,
            const float* __restrict__ kc, const float* __restrict__ kr,
            const float* __restrict__ sc, const float* __restrict__ sr,
            const double* __restrict__ rsub, int words, uint32_t* __restrict__ mask, int prof,
            int max_pairs, int task_words, int near, int64_t rsub_stride) {
  extern __shared__ float4 sm4[];
  __shared__ unsigned ubits_all[PLAN_WARPS][32], wbits_all[PLAN_WARPS][32];
  // positions of set bits, written by the lanes that hold them: the failing tiles of a chunk, the
  // ones (a) left open, and the open sub-balls of a pair of tiles (finding the n-th set bit of a
  // mask with __fns, a software loop, for every test took most of this kernel's time)
  __shared__ uint8_t fail_all[PLAN_WARPS][32], open_all[PLAN_WARPS][32];
  __shared__ uint8_t ulist_all[PLAN_WARPS][8], wlist_all[PLAN_WARPS][32];
  __shared__ double reach_all[PLAN_WARPS][4];
  const int lane = lane_id(), wib = warp_id();
  const int n4 = dp / 4;
  float4* qball = sm4 + wib * (9 * n4);          // [0]: tile, [1..8]: sub-balls
  unsigned* ubits = ubits_all[wib];
  unsigned* wbits = wbits_all[wib];
  uint8_t *fails = fail_all[wib], *opens = open_all[wib];
  uint8_t *ulist = ulist_all[wib], *wlist = wlist_all[wib];
  double* reach = reach_all[wib];
  const unsigned below = (1u << lane) - 1u;
  const float4* kc4 = reinterpret_cast<const float4*>(kc);     // interleaved
  const float4* sc4 = reinterpret_cast<const float4*>(sc);     // interleaved
  const double f = op_scale(prec, ctl);
  const int64_t warps = int64_t(gridDim.x) * PLAN_WARPS;
  const int nv = 2 * max(1, bn / SUB);          // key sub-balls per key tile
  long long nvis = 0, ntot = 0, nl1 = 0, npt = 0, npr = 0;
  // tasks = (query tile, block of task_words mask words): the level-2 work of a query tile varies
  // widely, so whole tiles per warp would leave most SMs idle behind the slowest few
  const int nblk = (words + task_words - 1) / task_words;
  const int64_t ntasks = n_items * nblk;
  // consecutive warps take consecutive query tiles of the same key-tile block, so the key-side
  // centres they read are shared through L1
  for (int64_t task = int64_t(blockIdx.x) * PLAN_WARPS + wib; task < ntasks; task += warps) {
    const int wblk = int(task / n_items);
    const int64_t it = task - int64_t(wblk) * n_items;
    const WorkItem w = items[it];
    const int64_t qt = w.qrow0 / QTILE;          // 128-row tile of packed rows
    const int64_t sb0 = int64_t(w.qrow0) / SUB;  // its first 32-row block
    __syncwarp();
    for (int t = lane; t < n4; t += 32)
      qball[t] = reinterpret_cast<const float4*>(qc)[qt * n4 + t];
    for (int x = lane; x < 8 * n4; x += 32) {       // 8 consecutive balls: 128-byte runs
      const int t = x >> 3, u = x & 7;
      qball[(1 + u) * n4 + t] = sc4[inter_at(2 * sb0 + u, n4) + int64_t(t) * INTER];
    }
    __syncwarp();
    const float rq = qr[qt];
    // the reach of each 32-row block and of the whole tile
    if (lane < 4)                                          // rsub is >= 0 or +inf
      reach[lane] = ball_reach(rsub[w.pad0 * rsub_stride + sb0 + lane], f);
    __syncwarp();
    const double reach_q = fmax(fmax(reach[0], reach[1]), fmax(reach[2], reach[3]));
    const int nkt = (w.nkeys + bn - 1) / bn;
    const int diag = (w.qrow0 - w.key0) / bn;
    // near tiles, which the scan visits anyway (near < 0: none, the queries are not among the keys)
    const int lo = max(0, diag - near), hi = min(nkt - 1, diag + near);
    uint32_t* out = mask + it * int64_t(words);
    const int wend = min(words, (wblk + 1) * task_words);
    for (int base = wblk * task_words * 32; base < wend * 32; base += 32) {
      const int kt = base + lane;
      bool l1 = false;                           // not separated at level 1
      bool deep = false;                         // ... and visited without level 2
      if (kt < nkt && (kt < lo || kt > hi)) {
        const int64_t g = (int64_t(w.key0) + int64_t(kt) * bn) / 256;
        const float d2 = ball_d2<1, INTER>(qball, kc4 + inter_at(g, n4), n4);
        l1 = !apart(d2, rq, kr[g], reach_q, d);
        // a key tile whose centre lies within the rows' reach of the query tile's shares its
        // cluster: level 2 would find open sub-balls (a visit it could have saved costs time only;
        // at 1.3M x 50 the visits are the same 2.88 M, and level 2 tests half the pairs)
        deep = l1 && double(d2) <= reach_q * reach_q;
        l1 = l1 && !deep;
      }
      const uint32_t fm = __ballot_sync(FULL, l1);
      uint32_t bits = __ballot_sync(FULL, deep);
      if (fm) {
        const int nf = __popc(fm);
        nl1 += nf;
        ubits[lane] = 0u;
        wbits[lane] = 0u;
        if (l1) fails[__popc(fm & below)] = uint8_t(lane);
        __syncwarp();
        // (a) query sub-ball u of failing tile i
        for (int x = lane; x < 8 * nf; x += 32) {
          const int i = x >> 3, u = x & 7;
          const int kti = base + fails[i];
          const int64_t g = (int64_t(w.key0) + int64_t(kti) * bn) / 256;
          if (!separated<1, INTER>(qball + (1 + u) * n4, sr[2 * sb0 + u], reach[u >> 1],
                                   kc4 + inter_at(g, n4), kr[g], n4, d))
            atomicOr(&ubits[i], 1u << u);
        }
        __syncwarp();
        // (b) key sub-ball v of failing tile i, only for the tiles (a) left open (a tile with no
        // open query sub-ball is skipped whatever (b) finds)
        const uint32_t fo = __ballot_sync(FULL, lane < nf && ubits[lane] != 0u);
        const int no = __popc(fo);
        if ((fo >> lane) & 1u) opens[__popc(fo & below)] = uint8_t(lane);
        __syncwarp();
        for (int x = lane; x < nv * no; x += 32) {
          const int io = x / nv, v = x - io * nv;
          const int i = opens[io];
          const int kti = base + fails[i];
          const int64_t kb0 = (int64_t(w.key0) + int64_t(kti) * bn) / SUB;
          const float rw = sr[2 * kb0 + v];
          if (rw >= 0.f && !separated<1, INTER>(qball, rq, reach_q,
                                                sc4 + inter_at(2 * kb0 + v, n4), rw, n4, d))
            atomicOr(&wbits[i], 1u << v);
        }
        __syncwarp();
        for (int i = 0; i < nf; ++i) {
          const uint32_t ub = ubits[i], wb = wbits[i];
          if (!ub || !wb) continue;                 // warp-uniform
          const int kti = base + fails[i];
          const int64_t kb0 = (int64_t(w.key0) + int64_t(kti) * bn) / SUB;
          const int nu = __popc(ub), npair = nu * __popc(wb);
          // many overlapping sub-ball pairs: the tiles share a cluster, and testing every pair
          // would almost always end in a visit anyway
          if (npair > max_pairs) {
            bits |= 1u << (kti - base);
            continue;
          }
          ++npt;
          npr += npair;
          __syncwarp();                             // the previous tile's lists are read
          if (lane < 8 && ((ub >> lane) & 1u)) ulist[__popc(ub & below)] = uint8_t(lane);
          if ((wb >> lane) & 1u) wlist[__popc(wb & below)] = uint8_t(lane);
          __syncwarp();
          bool hit = false;
          for (int pr = lane; pr < npair && !hit; pr += 32) {
            const int u = ulist[pr % nu], vv = wlist[pr / nu];
            hit = !separated<1, INTER>(qball + (1 + u) * n4, sr[2 * sb0 + u], reach[u >> 1],
                                       sc4 + inter_at(2 * kb0 + vv, n4), sr[2 * kb0 + vv], n4, d);
          }
          if (__any_sync(FULL, hit)) bits |= 1u << (kti - base);
        }
      }
      if (lane == 0) {
        out[base >> 5] = bits;
        nvis += __popc(bits);
      }
    }
    if (wblk == 0) ntot += nkt - (hi - lo + 1);
  }
  if (prof && lane == 0) {
    atomicAdd(&g_prune_tiles[0], (unsigned long long)nvis);
    atomicAdd(&g_prune_tiles[1], (unsigned long long)ntot);
    atomicAdd(&g_prune_tiles[2], (unsigned long long)nl1);
    atomicAdd(&g_prune_tiles[3], (unsigned long long)npt);
    atomicAdd(&g_prune_tiles[4], (unsigned long long)npr);
  }
}


// Point test of the kept pairs, one block per (256-key tile, item slice): a key tile whose bounding
// ball is wide (cells of two clusters, or outliers spread over the whole sample) fails the ball
// tests for almost every query tile even when no key of it is near.  Here every key is a ball of
// radius 0: the pair is skipped when every key y satisfies |c_Q − y| − r_Q = L > 0 and
// f²·L² > R_Q (c_Q, r_Q the query tile's ball, R_Q the largest R of its rows), the plan's own
// separation rule.  The tile's keys are staged once in shared memory, dimension-major (a warp's
// 32 keys of one dimension hit 32 banks); the query tiles that kept the tile are listed, and each
// warp takes whole query tiles from the list: its lanes test 8 keys each and stop at the first key
// that is not separated.  A pair every key clears has its bit taken out of the mask.
constexpr int POINT_T = 256;
constexpr int POINT_SLICES = 2;    // item slices per key tile (the long lists of outlier tiles)
constexpr int POINT_LIST = 2048;   // listed query tiles per round
__global__ void __launch_bounds__(POINT_T)
point_test_kernel(const float* __restrict__ X, int d, int dp, const int32_t* __restrict__ perm,
                  const WorkItem* __restrict__ items, int64_t n_items, int bn, int words,
                  const Ctl* ctl, int prec, const float* __restrict__ qc,
                  const float* __restrict__ qr, const double* __restrict__ rsub,
                  uint32_t* __restrict__ mask, int64_t nkt_all, int prof) {
  extern __shared__ float ys[];                       // [d][256] this tile's keys
  __shared__ int32_t list[POINT_LIST];
  __shared__ int nlist, next;
  __shared__ unsigned pad_bits[256 / 32];             // keys that are padding rows
  const int tid = threadIdx.x, lane = lane_id(), wib = warp_id();
  constexpr int NW = POINT_T / 32;
  const double f = op_scale(prec, ctl);
  const double f2 = f * f;
  const double shrink = 1.0 - double(d + 8) * 0x1p-23;
  long long cleared = 0;
  if (tid < 256 / 32) pad_bits[tid] = 0u;
  for (int64_t gb = blockIdx.x; gb < nkt_all * POINT_SLICES; gb += gridDim.x) {   // block-uniform
    const int64_t g = gb / POINT_SLICES;
    const int slice = int(gb - g * POINT_SLICES);
    const int64_t p0 = g * 256;
    __syncthreads();                                   // the previous tile's keys are done with
    // keys: a warp per row (coalesced), dimension-major in shared memory
    for (int r = wib; r < 256; r += NW) {
      const int32_t i = perm[p0 + r];
      for (int t = lane; t < d; t += 32) ys[t * 256 + r] = i < 0 ? 0.f : X[int64_t(i) * d + t];
      const unsigned pb = __ballot_sync(FULL, i < 0);  // warp-uniform i: all lanes agree
      if (lane == 0) atomicOr(&pad_bits[r >> 5], (pb ? 1u : 0u) << (r & 31));
    }
    for (int64_t base = slice; base < n_items; base += int64_t(POINT_SLICES) * POINT_LIST) {
      __syncthreads();
      if (tid == 0) { nlist = 0; next = 0; }
      __syncthreads();
      for (int j = tid; j < POINT_LIST; j += POINT_T) {
        const int64_t it = base + int64_t(j) * POINT_SLICES;
        if (it < n_items) {
          const WorkItem w = items[it];
          const int64_t rel = p0 - w.key0;
          if (rel >= 0 && rel < w.nkeys) {
            const int kt = int(rel / bn);
            if (mask[it * words + (kt >> 5)] & (1u << (kt & 31)))
              list[atomicAdd(&nlist, 1)] = int32_t(it);
          }
        }
      }
      __syncthreads();
      const int nl = nlist;
      for (;;) {                                       // warp-uniform: a query tile per warp
        int k = 0;
        if (lane == 0) k = atomicAdd(&next, 1);
        k = __shfl_sync(FULL, k, 0);
        if (k >= nl) break;
        const int32_t it = list[k];
        const WorkItem w = items[it];
        const int64_t qt = w.qrow0 / QTILE, sb0 = w.qrow0 / SUB;
        double R = 0.0;
        for (int j = 0; j < 4; ++j) R = fmax(R, rsub[sb0 + j]);
        const float rq = qr[qt];
        if (!(rq >= 0.f) || !(R < 1e300)) continue;     // nothing provable for this tile
        const float* c = qc + qt * dp;
        bool all = true;
        for (int kk = 0; kk < 8 && all; ++kk) {          // keys lane + 32·kk
          const int key = lane + 32 * kk;
          bool sep = true;
          if (!((pad_bits[key >> 5] >> (key & 31)) & 1u)) {
            float acc = 0.f;
            for (int t = 0; t < d; ++t) {
              const float u = c[t] - ys[t * 256 + key];
              acc = fmaf(u, u, acc);
            }
            const double L = sqrt(fmax(0.0, double(acc) * shrink - F32_SQ_FLOOR)) - double(rq);
            sep = L > 0.0 && f2 * L * L > R * (1.0 + 1e-9);
          }
          all = __all_sync(FULL, sep);
        }
        if (all && lane == 0) {
          const int kt = int((p0 - w.key0) / bn);
          atomicAnd(&mask[int64_t(it) * words + (kt >> 5)], ~(1u << (kt & 31)));
          ++cleared;
        }
      }
    }
    __syncthreads();
    if (tid < 256 / 32) pad_bits[tid] = 0u;            // for the next tile
  }
  if (prof && cleared) atomicAdd(&g_prune_tiles[0], (unsigned long long)(-cleared));
}

// Visit mask of every work item of the refine pass (the rows whose one-term certificate failed,
// re-scanned with the three-term split).  A refine item holds up to 128 such rows from anywhere in
// their sample; its mask is the union of its rows' query-tile masks and near tiles.  This stays
// exact for the refine values v3 if each row's
// one-term error bound, in the unscaled space, covers the three-term one (eps1 >= f²·eps3): the
// skipped keys have v > (thr + 3·eps1)/f², the near-pass keys (never skipped) v <= (thr + eps1)/f²,
// so every skipped key's v3 lies above the refine threshold.  An item with a row where that fails
// scans every key tile.
__global__ void refine_mask_kernel(const WorkItem* __restrict__ items3,
                                   const int32_t* __restrict__ n_items3,
                                   const int32_t* __restrict__ qmap,
                                   const SegDesc* __restrict__ seg, int nseg,
                                   const uint32_t* __restrict__ mask, int words, int bn,
                                   const QStat* __restrict__ qs, const KeyMax* __restrict__ km,
                                   const QStat* __restrict__ qs3, const KeyMax* __restrict__ km3,
                                   const Ctl* __restrict__ ctl, int prec, int kmma, int kmma3,
                                   int d, uint32_t* __restrict__ mask3) {
  const int lane = lane_id();
  const int64_t warps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  const int nitems = *n_items3;
  const double f = op_scale(prec, ctl);
  const KeyMax K1 = *km, K3 = *km3;
  for (int64_t r = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5; r < nitems; r += warps) {
    const WorkItem w = items3[r];
    const int nkt = (w.nkeys + bn - 1) / bn;
    bool ok = true;
    for (int j = lane; j < w.nq; j += 32) {
      const int32_t p = qmap[w.qrow0 + j];
      ok = ok && cert_eps(qs[p], K1, prec, kmma, d) >= f * f * cert_eps(qs3[p], K3, PREC_BF16X3, kmma3, d);
    }
    ok = __all_sync(FULL, ok);
    uint32_t* out = mask3 + r * int64_t(words);
    for (int wi = lane; wi < words; wi += 32) {
      uint32_t acc = 0u;
      if (!ok) {
        acc = 0xffffffffu;
      } else {
        for (int j = 0; j < w.nq; ++j) {
          const int32_t p = qmap[w.qrow0 + j];
          const SegDesc sg = seg[find_seg(seg, nseg, p)];
          const int64_t mi = sg.tile0 + (p - sg.poff) / QTILE;       // its query tile's item
          acc |= mask[mi * words + wi];
          const int dj = int(((p - sg.poff) / QTILE * QTILE) / bn);    // that tile's near range
          const int l0 = max(0, dj - 2) - wi * 32, h0 = min(nkt - 1, dj + 2) - wi * 32;
          for (int b = max(0, l0); b <= min(31, h0); ++b) acc |= 1u << b;
        }
      }
      // never beyond the sample (refine walks have no near phase: the item's own near tiles
      // stay in the mask)
      for (int b = 0; b < 32; ++b) {
        const int kt = wi * 32 + b;
        if (kt >= nkt) acc &= ~(1u << b);
      }
      out[wi] = acc;
    }
  }
}

// Seeds of the refine pass: the main scan kept k' keys with one-term values at or below thr, so
// their true values are at most (thr + eps1)/f² and their three-term values at most eps3 more: the
// row's k'-th three-term value does not exceed that, and the pass need not keep anything above.
// Without it each of a row's eight parts fills a list anew (18 insertions per cell of the sample,
// now one): graphs of 200,000 cells 8.2 -> 7.55 ms, of 1.3 M 63.1 -> 61.5.
// (A row of a long item has its merged k'-th value in seed and excl.x = -1: its threshold can be
// a part's, which fewer than k' keys may reach.)
__global__ void refine_seed_kernel(const int32_t* __restrict__ qmap,
                                   const int32_t* __restrict__ n_rows,
                                   const int32_t* __restrict__ perm,
                                   const float* __restrict__ cand_thr,
                                   const float* __restrict__ seed, const int4* __restrict__ excl,
                                   const QStat* __restrict__ qs, const KeyMax* __restrict__ km,
                                   const QStat* __restrict__ qs3, const KeyMax* __restrict__ km3,
                                   const Ctl* __restrict__ ctl, int prec, int kmma, int kmma3,
                                   int d, float* __restrict__ seed3) {
  const int64_t n = *n_rows;
  const double f = op_scale(prec, ctl), f3 = op_scale(PREC_BF16X3, ctl);
  const KeyMax K1 = *km, K3 = *km3;
  for (int64_t q = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; q < n;
       q += int64_t(gridDim.x) * blockDim.x) {
    const int32_t p = qmap[q];
    const double t = excl[p].x == -1 ? seed[p] : cand_thr[perm[p]];
    const double e1 = cert_eps(qs[p], K1, prec, kmma, d);
    const double e3 = cert_eps(qs3[p], K3, PREC_BF16X3, kmma3, d);
    const double s = (t + e1) * (f3 / f) * (f3 / f) + e3;
    seed3[q] = s < 1e30 ? nextafterf(__double2float_ru(s), F_INF) : F_INF;   // NaN: no seed
  }
}

// Merge of a split refine pass: warp per refine row; the S·k' entries of its S work items, the k'
// smallest kept (ties: lower lane, then lower slot).  The threshold is the k'-th smallest or, if
// that is less, the work items' smallest (their seed, with which a list may stay short): every key
// that a work item dropped is at least its threshold.
__global__ void refine_merge_kernel(const WorkItem* __restrict__ items3,
                                    const int32_t* __restrict__ n_items3,
                                    const Ctl* __restrict__ ctl, const int32_t* __restrict__ qmap,
                                    const int32_t* __restrict__ perm,
                                    const int2* __restrict__ part,
                                    const float* __restrict__ part_thr, int kprime,
                                    int32_t* __restrict__ cand_idx, float* __restrict__ cand_thr) {
  const int S = ctl->refine_split;
  if (S <= 1) return;
  const int lane = lane_id();
  const int nitems = *n_items3;
  const int64_t warps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  const int per = (S * kprime + 31) / 32;              // entries per lane (<= 16)
  for (int64_t x = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5;
       x < int64_t(nitems) * QTILE; x += warps) {
    const int r = int(x / QTILE), j = int(x % QTILE);
    const WorkItem w = items3[r];
    if (j >= w.nq) continue;                          // warp-uniform
    float v[16];
    int id[16];
#pragma unroll
    for (int t = 0; t < 16; ++t) {
      v[t] = F_INF;
      id[t] = -1;
      const int e = lane + 32 * t;
      if (t < per && e < S * kprime) {
        const int s = e / kprime, slot = e - s * kprime;
        const int2 pe = part[((int64_t(r) * S + s) * QTILE + j) * kprime + slot];
        if (pe.y >= 0) { v[t] = __int_as_float(pe.x); id[t] = pe.y; }
      }
    }
    const int64_t orow = perm[qmap[w.qrow0 + j]];
    float thr = lane < S ? part_thr[(int64_t(r) * S + lane) * QTILE + j] : F_INF;   // S <= 32
    for (int o = 16; o > 0; o >>= 1) thr = fminf(thr, __shfl_xor_sync(FULL, thr, o));
    float kth = F_INF;
    for (int o = 0; o < kprime; ++o) {
      float bv = F_INF;
      int bt = 16;
#pragma unroll
      for (int t = 0; t < 16; ++t)
        if (v[t] < bv) { bv = v[t]; bt = t; }
      // warp argmin of (value, lane)
      float mv = bv;
      int ml = lane;
      for (int off = 16; off > 0; off >>= 1) {
        const float ov = __shfl_xor_sync(FULL, mv, off);
        const int ol = __shfl_xor_sync(FULL, ml, off);
        if (ov < mv || (ov == mv && ol < ml)) { mv = ov; ml = ol; }
      }
      int out = -1;
      if (lane == ml && bt < 16) {
#pragma unroll
        for (int t = 0; t < 16; ++t)
          if (t == bt) { out = id[t]; v[t] = F_INF; }
      }
      out = __shfl_sync(FULL, out, ml);
      if (lane == 0) cand_idx[orow * kprime + o] = mv < F_INF ? out : -1;
      kth = mv;
    }
    if (lane == 0) cand_thr[orow] = fminf(kth, thr);
  }
}

// ---- sorted visit lists of the main scan ----

// |z|² + 3·eps of every packed row of the final layout: the part of the row's radius
// R = threshold + roff that stays fixed while the scan lowers the threshold (as R is formed from
// the near pass's threshold in row_radius_kernel)
__global__ void row_offset_kernel(const int32_t* __restrict__ perm, int64_t npacked,
                                  const QStat* __restrict__ qs, const KeyMax* __restrict__ km,
                                  int prec, int kmma, int d, double* __restrict__ roff) {
  for (int64_t p = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; p < npacked;
       p += int64_t(gridDim.x) * blockDim.x) {
    if (perm[p] < 0) { roff[p] = 0.0; continue; }
    const QStat q = qs[p];
    roff[p] = q.sq + 3.0 * cert_eps(q, *km, prec, kmma, d);
  }
}

// kept far tiles per work item (warp per item)
__global__ void visit_count_kernel(const uint32_t* __restrict__ mask, int64_t n_items, int words,
                                   int32_t* __restrict__ cnt) {
  const int lane = lane_id();
  const int64_t warps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t it = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5; it < n_items;
       it += warps) {
    int c = 0;
    for (int wi = lane; wi < words; wi += 32) c += __popc(mask[it * words + wi]);
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(FULL, c, o);
    if (lane == 0) cnt[it] = c;
  }
}

// Claim order of the main scan's work items, costliest first.  Cost = the far tiles the plan kept
// (every item also scans its few near tiles), in COST_BUCKETS buckets of 2^shift tiles.  The
// persistent CTAs claim items in this order, so the long items (rows whose radius reaches many
// key tiles) start first instead of ending the launch on a few SMs.
constexpr int COST_BUCKETS = 256;
__global__ void cost_hist_kernel(const int32_t* __restrict__ cnt, int64_t n_items, int shift,
                                 int32_t* __restrict__ hist) {
  __shared__ int32_t h[COST_BUCKETS];
  for (int b = threadIdx.x; b < COST_BUCKETS; b += blockDim.x) h[b] = 0;
  __syncthreads();
  for (int64_t it = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; it < n_items;
       it += int64_t(gridDim.x) * blockDim.x)
    atomicAdd(&h[min(COST_BUCKETS - 1, cnt[it] >> shift)], 1);
  __syncthreads();
  for (int b = threadIdx.x; b < COST_BUCKETS; b += blockDim.x)
    if (h[b]) atomicAdd(&hist[b], h[b]);
}
// one block of COST_BUCKETS threads: hist[b] := items in buckets above b (descending offsets)
__global__ void cost_offsets_kernel(int32_t* __restrict__ hist) {
  __shared__ int32_t h[COST_BUCKETS];
  const int b = threadIdx.x;
  h[b] = hist[b];
  __syncthreads();
  int32_t above = 0;
  for (int j = b + 1; j < COST_BUCKETS; ++j) above += h[j];
  hist[b] = above;
}
__global__ void cost_scatter_kernel(const int32_t* __restrict__ cnt, int64_t n_items, int shift,
                                    int32_t* __restrict__ off, int32_t* __restrict__ order) {
  for (int64_t it = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; it < n_items;
       it += int64_t(gridDim.x) * blockDim.x) {
    const int b = min(COST_BUCKETS - 1, cnt[it] >> shift);
    order[atomicAdd(&off[b], 1)] = int32_t(it);
  }
}

// The long items (a tile of outliers visits most key tiles and inserts into every row at other
// times than its neighbours) would each keep one CTA busy after the others have run out of items.
// Those whose cost is above LONG_SHARE of a CTA's share of all are scanned in LONG_SPLIT parts by
// different CTAs, and their lists merged.  100,000 cells: twenty tiles took 2.0 to 2.6 ms each
// where the CTAs' mean was 0.94; graph 6.0 -> 4.9 ms, of 200,000 cells 8.9 -> 8.2.  Parts insert
// more than the whole item, so only what would outlast a mean CTA is split: at shares of 0.5 and
// 0.25 100,000 cells take 5.2 and 5.6 ms, 1.3 M 63 and 73 (1.0: 63).  The parts' lists hold 32 of
// k' = 48: with 24 the 200,000 cells take 8.5 ms (more rows left to the refine pass), with 48 the
// 100,000 take 0.2 ms more.
// With fewer than two items per CTA a CTA's share falls below the items' mean, and items like all the
// others would count as long: of 31,382 uniform cells (246 items, 296 CTAs) every one was, with five
// times the insertions.  So a long item also costs LONG_TIMES the mean: cohorts of 43,947 cells in
// seven samples 3.44 -> 2.30 ms, of 24,866 in four 2.42 -> 1.70.
constexpr double LONG_SHARE = 1.0, LONG_TIMES = 2.0;
constexpr int LONG_NEAR = 5;          // near tiles an item scans besides
constexpr int LONG_T = 1024;
__global__ void __launch_bounds__(LONG_T)
long_plan_kernel(const int32_t* __restrict__ cnt, int64_t n_items, int shift, int n_ctas,
                 int max_long, const int32_t* __restrict__ order, int32_t* __restrict__ claim,
                 Ctl* __restrict__ ctl, int prof) {
  __shared__ unsigned long long total;
  __shared__ int n_long;
  if (threadIdx.x == 0) { total = 0; n_long = 0; }
  __syncthreads();
  unsigned long long t = 0;
  for (int64_t i = threadIdx.x; i < n_items; i += LONG_T) t += cnt[i] + LONG_NEAR;
  atomicAdd(&total, t);
  __syncthreads();
  // whole buckets of the claim order, so that the long items are its first ones
  const double cut = double(total) * fmax(LONG_SHARE / n_ctas, LONG_TIMES / double(n_items));
  const int bucket = int(fmin(cut, 1e9)) >> shift;
  int m = 0;
  for (int64_t i = threadIdx.x; i < n_items; i += LONG_T)
    m += min(COST_BUCKETS - 1, cnt[i] >> shift) > bucket ? 1 : 0;
  atomicAdd(&n_long, m);
  __syncthreads();
  const int64_t n = min(n_long, max_long), parts = n * LONG_SPLIT;
  for (int64_t j = threadIdx.x; j < n_items - n + parts; j += LONG_T)
    claim[j] = j < parts ? LONG_FLAG | int32_t(j) : order[j - parts + n];
  if (threadIdx.x == 0) {
    ctl->n_long = int32_t(n);
    ctl->n_items_main = int32_t(n_items - n + parts);
    if (prof) atomicAdd(&g_prune_tiles[5], (unsigned long long)n);
  }
}

// Merge of the long items' parts: warp per row; the near pass's list (its keys are not offered
// again) and the parts' kper entries each, the k' smallest kept.  A key that none of them holds
// was at or above its part's threshold or, in the near pass, the near list's k'-th value, which
// the merged k'-th value does not exceed.
__global__ void long_merge_kernel(const WorkItem* __restrict__ items, const Ctl* __restrict__ ctl,
                                  const int32_t* __restrict__ order,
                                  const int32_t* __restrict__ perm,
                                  const int2* __restrict__ part,
                                  const float* __restrict__ part_thr,
                                  const float* __restrict__ near_val, int kprime, int kper,
                                  int32_t* __restrict__ cand_idx, float* __restrict__ cand_thr,
                                  float* __restrict__ seed, int4* __restrict__ excl) {
  const int lane = lane_id();
  const int64_t rows = int64_t(ctl->n_long) * QTILE;
  const int64_t warps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  const int total = kprime + LONG_SPLIT * kper;        // <= 9 * 64
  for (int64_t x = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5; x < rows; x += warps) {
    const int64_t r = x / QTILE;
    const int j = int(x % QTILE);
    const WorkItem w = items[order[r]];
    if (j >= w.nq) continue;                           // warp-uniform
    const int64_t orow = perm[w.qrow0 + j];
    float v[18];
    int id[18];
#pragma unroll
    for (int t = 0; t < 18; ++t) {
      v[t] = F_INF;
      id[t] = -1;
      const int e = lane + 32 * t;
      if (e < kprime) {
        const int c = cand_idx[orow * kprime + e];
        if (c >= 0) { v[t] = near_val[orow * kprime + e]; id[t] = c; }
      } else if (e < total) {
        const int s = (e - kprime) / kper, slot = (e - kprime) % kper;
        const int2 pe = part[((r * LONG_SPLIT + s) * QTILE + j) * kprime + slot];
        if (pe.y >= 0) { v[t] = __int_as_float(pe.x); id[t] = pe.y; }
      }
    }
    float thr = lane < LONG_SPLIT ? part_thr[(r * LONG_SPLIT + lane) * QTILE + j] : F_INF;
    for (int o = 16; o > 0; o >>= 1) thr = fminf(thr, __shfl_xor_sync(FULL, thr, o));
    __syncwarp();                                      // the list is read before it is written
    float kth = F_INF;
    for (int o = 0; o < kprime; ++o) {
      float bv = F_INF;
      int bt = 18;
#pragma unroll
      for (int t = 0; t < 18; ++t)
        if (v[t] < bv) { bv = v[t]; bt = t; }
      float mv = bv;                                   // warp argmin of (value, lane)
      int ml = lane;
      for (int off = 16; off > 0; off >>= 1) {
        const float ov = __shfl_xor_sync(FULL, mv, off);
        const int ol = __shfl_xor_sync(FULL, ml, off);
        if (ov < mv || (ov == mv && ol < ml)) { mv = ov; ml = ol; }
      }
      int out = -1;
      if (lane == ml && bt < 18) {
#pragma unroll
        for (int t = 0; t < 18; ++t)
          if (t == bt) { out = id[t]; v[t] = F_INF; }
      }
      out = __shfl_sync(FULL, out, ml);
      if (lane == 0) cand_idx[orow * kprime + o] = mv < F_INF ? out : -1;
      kth = mv;
    }
    if (lane == 0) {
      cand_thr[orow] = fminf(kth, thr);
      seed[w.qrow0 + j] = fminf(kth, seed[w.qrow0 + j]);   // for the refine pass (refine_seed)
      excl[w.qrow0 + j].x = -1;
    }
  }
}

constexpr int VO_T = 256;            // threads per block of the order kernel
constexpr int VO_SORT_MAX = 8192;    // longest list sorted (longer ones keep tile order)

// One block per work item: its kept far tiles (the set bits of its mask) in order of the distance
// between the 128-row query tile's ball centre and the 256-row key ball's centre (ties by tile):
// nearest first, so the rows' thresholds fall early and later tiles rarely insert.  Each entry
// carries a stop bound: the smallest need over it and every later entry, need = f²·L²,
// L = |c_Q − c_K|·sqrt(1 − e) − r_Q − r_K (the float distance lowered by its rounding bound e as in
// separated()), rounded down, 0 when L <= 0; need <= f²·|x − y|² for every row x of the tile and
// key y of the key tile (unscaled coordinates, f = the operand scale), so once an entry's bound
// exceeds every row's radius, no later tile can give a row a candidate.
__global__ void __launch_bounds__(VO_T)
visit_order_kernel(const WorkItem* __restrict__ items, int64_t n_items, int bn, int d, int dp,
                   const Ctl* __restrict__ ctl, int prec, const float* __restrict__ qc,
                   const float* __restrict__ qr, const float* __restrict__ kc,
                   const float* __restrict__ kr, const uint32_t* __restrict__ mask, int words,
                   const int64_t* __restrict__ voff, int64_t cap,
                   unsigned long long* __restrict__ vlist, int32_t* __restrict__ ok_flag) {
  extern __shared__ unsigned long long vo_keys[];                 // [VO_SORT_MAX] dist | pos
  int32_t* vo_kt = reinterpret_cast<int32_t*>(vo_keys + VO_SORT_MAX);   // [VO_SORT_MAX]
  float* vo_need = reinterpret_cast<float*>(vo_kt + VO_SORT_MAX);       // [VO_SORT_MAX]
  float* qcen = vo_need + VO_SORT_MAX;                                  // [dp]
  int32_t* wpre = reinterpret_cast<int32_t*>(qcen + dp);                // [words + 1]
  const bool fits = voff[n_items] <= cap;
  if (blockIdx.x == 0 && threadIdx.x == 0) *ok_flag = fits ? 1 : 0;
  if (!fits) return;
  const double f = op_scale(prec, ctl);
  const double f2 = f * f;
  const double e = double(d + 8) * 0x1p-23;
  const int n4 = dp / 4;
  for (int64_t it = blockIdx.x; it < n_items; it += gridDim.x) {
    const WorkItem w = items[it];
    const int64_t o = voff[it];
    const int c = int(voff[it + 1] - o);
    if (c == 0) continue;                                         // block-uniform
    const int64_t qt = w.qrow0 / QTILE;
    __syncthreads();
    for (int t = threadIdx.x; t < dp; t += VO_T) qcen[t] = qc[qt * dp + t];
    // exclusive prefix of the words' bit counts (one thread; words is small)
    if (threadIdx.x == 0) {
      int a = 0;
      for (int wi = 0; wi < words; ++wi) { wpre[wi] = a; a += __popc(mask[it * words + wi]); }
      wpre[words] = a;
    }
    __syncthreads();
    const float rq = qr[qt];
    const bool sorted = c <= VO_SORT_MAX;
    for (int wi = threadIdx.x; wi < words; wi += VO_T) {
      uint32_t bits = mask[it * words + wi];
      int pos = wpre[wi];
      while (bits) {
        const int b = __ffs(bits) - 1;
        bits &= bits - 1u;
        const int kt = wi * 32 + b;
        if (!sorted) {                  // tile order, no stop bound (-inf never ends a walk)
          vlist[o + pos] = (static_cast<unsigned long long>(__float_as_uint(-F_INF)) << 32) |
                           uint32_t(kt);
          ++pos;
          continue;
        }
        const int64_t g = (int64_t(w.key0) + int64_t(kt) * bn) / 256;
        const float rk = kr[g];
        float dist = 0.f, need = F_INF;
        if (rq >= 0.f && rk >= 0.f) {
          const float4* a4 = reinterpret_cast<const float4*>(qcen);
          const float4* b4 = reinterpret_cast<const float4*>(kc) + inter_at(g, n4);
          float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
          for (int t = 0; t < n4; ++t) {
            const float4 x = a4[t], y = b4[t * INTER];
            const float e0 = x.x - y.x, e1 = x.y - y.y, e2 = x.z - y.z, e3 = x.w - y.w;
            s0 = fmaf(e0, e0, s0);
            s1 = fmaf(e1, e1, s1);
            s2 = fmaf(e2, e2, s2);
            s3 = fmaf(e3, e3, s3);
          }
          const float sum = (s0 + s1) + (s2 + s3);
          dist = sum;
          const double L = sqrt(fmax(0.0, double(sum) * (1.0 - e) - F32_SQ_FLOOR)) -
                           double(rq) - double(rk);
          need = L > 0.0 ? __double2float_rd(f2 * L * L * (1.0 - 1e-12)) : 0.f;
        } else {
          dist = F_INF;                 // a ball without rows: no candidate, last
        }
        vo_kt[pos] = kt;
        vo_need[pos] = need;
        vo_keys[pos] = (static_cast<unsigned long long>(__float_as_uint(dist)) << 32) |
                       uint32_t(pos);
        ++pos;
      }
    }
    if (!sorted) continue;                                        // block-uniform
    int P2 = 1;
    while (P2 < c) P2 <<= 1;
    __syncthreads();
    for (int t = c + threadIdx.x; t < P2; t += VO_T) vo_keys[t] = ~0ull;
    __syncthreads();
    // dist >= 0, so the float bits order as the values do; pos breaks ties in tile order
    for (int kk = 2; kk <= P2; kk <<= 1) {
      for (int jj = kk >> 1; jj > 0; jj >>= 1) {
        for (int t = threadIdx.x; t < P2; t += VO_T) {
          const int u = t ^ jj;
          if (u > t) {
            const unsigned long long a = vo_keys[t], b = vo_keys[u];
            const bool up = (t & kk) == 0;
            if ((a > b) == up) { vo_keys[t] = b; vo_keys[u] = a; }
          }
        }
        __syncthreads();
      }
    }
    // suffix minimum of the stop bounds along the sorted order (one thread), then the entries
    if (threadIdx.x == 0) {
      float m = F_INF;
      for (int j = c - 1; j >= 0; --j) {
        const int p = int(uint32_t(vo_keys[j]));
        m = fminf(m, vo_need[p]);
        vlist[o + j] = (static_cast<unsigned long long>(__float_as_uint(m)) << 32) |
                       uint32_t(vo_kt[p]);
      }
    }
  }
}

int grid_for(int64_t n) {
  return int(std::max<int64_t>(1, std::min<int64_t>(ceil_div(n, PR_T), int64_t(num_sms()) * 8)));
}

}  // namespace

int prune_mask_words(int64_t max_seg, int bn) {
  return int(ceil_div(ceil_div(max_seg, bn), 32));
}

namespace {
int plan_grid(int64_t n_items, int words, int& task_words) {
  const int64_t want = int64_t(num_sms()) * 6 * PLAN_WARPS * PLAN_TASKS;
  task_words = PLAN_WORDS_MAX;
  while (task_words > 1 && n_items * ceil_div(words, task_words) < want) task_words >>= 1;
  const int64_t ntasks = n_items * ceil_div(words, task_words);
  return int(std::max<int64_t>(1, std::min<int64_t>(ceil_div(ntasks, PLAN_WARPS),
                                                    int64_t(num_sms()) * 32)));
}

// ---- batch-balanced scans: queries in a region of their own behind the keys ----

// squared distance of every row to the mean of its 128-row tile (rows of no dense region are far)
__global__ void __launch_bounds__(PR_T)
tile_spread_kernel(const float* __restrict__ X, int d, const int32_t* __restrict__ perm,
                   int64_t ngroups, double* __restrict__ out) {
  constexpr int W = PR_T / 32, R = QTILE / W;
  __shared__ double part[W][MSC_MAX_D];
  __shared__ float c[MSC_MAX_D];
  __shared__ int cnts[W];
  const int lane = lane_id(), wib = warp_id();
  for (int64_t g = blockIdx.x; g < ngroups; g += gridDim.x) {
    const int64_t p0 = g * QTILE + wib * R;
    const int32_t my_i = lane < R ? perm[p0 + lane] : -1;
    double s[4] = {0, 0, 0, 0};
#pragma unroll 4
    for (int r = 0; r < R; ++r) {
      const int32_t i = __shfl_sync(FULL, my_i, r);
      if (i < 0) continue;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (lane + 32 * j < d) s[j] += X[int64_t(i) * d + lane + 32 * j];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (lane + 32 * j < d) part[wib][lane + 32 * j] = s[j];
    const unsigned have = __ballot_sync(FULL, my_i >= 0);
    if (lane == 0) cnts[wib] = __popc(have);
    __syncthreads();
    int cnt = 0;
    for (int w = 0; w < W; ++w) cnt += cnts[w];
    for (int t = threadIdx.x; t < d; t += PR_T) {
      double a = 0.0;
      for (int w = 0; w < W; ++w) a += part[w][t];
      c[t] = cnt ? float(a / cnt) : 0.f;
    }
    __syncthreads();
    for (int r = 0; r < R; r += 4) {
      const int rr = r + (lane >> 3);
      const int32_t i = __shfl_sync(FULL, my_i, rr);
      const double a = row_d2_8(X + int64_t(i < 0 ? 0 : i) * d, c, d, lane & 7);
      if ((lane & 7) == 0)
        out[p0 + rr] = i >= 0 ? a : __longlong_as_double(0x7ff8000000000000ll);
    }
  }
}

// stable partition of one sample: flagged rows first, then the others (leaf OUTLIER_LEAF)
__global__ void flag_partition_kernel(const int32_t* __restrict__ perm,
                                      const int32_t* __restrict__ leaf, int64_t n, int64_t npacked,
                                      const int32_t* __restrict__ reg,
                                      const int64_t* __restrict__ S, int32_t* __restrict__ perm2,
                                      int32_t* __restrict__ leaf2) {
  for (int64_t p = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; p < npacked;
       p += int64_t(gridDim.x) * blockDim.x) {
    const bool row = p < n;
    const int64_t pos = !row ? p : (reg[p] ? S[p] : S[n] + p - S[p]);
    perm2[pos] = perm[p];
    leaf2[pos] = row && !reg[p] ? OUTLIER_LEAF : leaf[p];
  }
}

// one bit per (query tile, batch) item: the batch's key tile whose ball centre is nearest
__global__ void nearest_tile_kernel(const WorkItem* __restrict__ items, int64_t n_items, int n4,
                                    const float* __restrict__ qc, const float* __restrict__ kc,
                                    const float* __restrict__ kr, int words,
                                    uint32_t* __restrict__ mask) {
  const int lane = lane_id();
  const float4* kc4 = reinterpret_cast<const float4*>(kc);
  const int64_t warps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t it = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5; it < n_items;
       it += warps) {
    const WorkItem w = items[it];
    const float4* q = reinterpret_cast<const float4*>(qc) + (w.qrow0 / QTILE) * int64_t(n4);
    const int nkt = (w.nkeys + 255) / 256;
    float best = F_INF;
    int at = 0;
    for (int kt = lane; kt < nkt; kt += 32) {
      const int64_t g = w.key0 / 256 + kt;
      if (kr[g] < 0.f) continue;
      const float d2 = ball_d2<1, INTER>(q, kc4 + inter_at(g, n4), n4);
      if (d2 < best) { best = d2; at = kt; }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const float od = __shfl_xor_sync(FULL, best, o);
      const int ok = __shfl_xor_sync(FULL, at, o);
      if (od < best || (od == best && ok < at)) { best = od; at = ok; }
    }
    for (int wi = lane; wi < words; wi += 32)
      mask[it * words + wi] = wi == (at >> 5) ? 1u << (at & 31) : 0u;
  }
}

// after the near pass: every (query, batch)'s radius R as in row_radius_kernel, its seed as in
// partition_kernel, and the largest R of each 32-row block of queries
__global__ void __launch_bounds__(PR_T)
query_radius_kernel(const int32_t* __restrict__ perm, int64_t p1, int64_t n, int nb,
                    const float* __restrict__ cand_thr, const QStat* __restrict__ qs,
                    const KeyMax* __restrict__ km, int prec, int kmma, int d, int64_t nqblk,
                    float* __restrict__ seed, double* __restrict__ rsub) {
  const int lane = lane_id();
  const int64_t warps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t x = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5; x < nqblk * nb;
       x += warps) {
    const int64_t b = x / nqblk, blk = x - b * nqblk, j = blk * 32 + lane;
    double r = 0.0;
    if (j < n) {
      const double thr = cand_thr[b * n + perm[p1 + j]];
      const QStat q = qs[p1 + j];
      const double eps = cert_eps(q, *km, prec, kmma, d);
      r = thr + q.sq + 3.0 * eps;
      if (!(r < 1e300)) r = __longlong_as_double(0x7ff0000000000000ll);
      const double t = thr + 2.0 * eps;
      seed[b * n + j] = t < 1e300 ? nextafterf(__double2float_ru(t), F_INF) : F_INF;
    }
    r = warp_max_d(r);
    if (lane == 0) rsub[b * nqblk + blk] = r;
  }
}
}  // namespace

int launch_order_outliers(const float* X, int d, const SegDesc* seg, int64_t n, int64_t npacked,
                          int32_t* perm, int32_t* leaf, const PruneWs& w, cudaStream_t st) {
  const int64_t ng = npacked / QTILE;
  const int grid = grid_for(npacked);
  tile_spread_kernel<<<int(std::min<int64_t>(ng, int64_t(num_sms()) * 32)), PR_T, 0, st>>>(
      X, d, perm, ng, w.rpos);
  MSC_LAUNCH_CHECK();
  sample_mean_partial_kernel<<<dim3(MEAN_CHUNKS, 1), PR_T, 0, st>>>(seg, 1, w.rpos, w.mean_part);
  MSC_LAUNCH_CHECK();
  sample_mean_final_kernel<<<1, 128, 0, st>>>(w.mean_part, 1, w.mean);
  MSC_LAUNCH_CHECK();
  regular_flag_kernel<<<grid, PR_T, 0, st>>>(perm, npacked, seg, 1, w.rpos, w.mean,
                                             OUTLIER_FACTOR, w.reg);
  MSC_LAUNCH_CHECK();
  MSC_TRY(scan_excl_i32(w.reg, n, w.S, w.scan_scratch, st));
  flag_partition_kernel<<<grid, PR_T, 0, st>>>(perm, leaf, n, npacked, w.reg, w.S, w.perm2,
                                               w.leaf2);
  MSC_LAUNCH_CHECK();
  MSC_CUDA_TRY(cudaMemcpyAsync(perm, w.perm2, sizeof(int32_t) * npacked, cudaMemcpyDeviceToDevice,
                               st));
  MSC_CUDA_TRY(cudaMemcpyAsync(leaf, w.leaf2, sizeof(int32_t) * npacked, cudaMemcpyDeviceToDevice,
                               st));
  return MSC_OK;
}

int launch_query_balls(const float* X, int d, int64_t npk, int64_t p1, int64_t nq,
                       const int32_t* perm, const int32_t* leaf, const double* zeros,
                       const PruneWs& w, cudaStream_t st) {
  const int dp = int(round_up(d, 4));
  const int64_t most = int64_t(num_sms()) * 32, nk = p1 / 256, ns = npk / SUB;
  group_ball_kernel<QTILE, false><<<int(std::min(nq, most)), PR_T, 0, st>>>(
      X, d, dp, perm + p1, nq, w.qc + (p1 / QTILE) * dp, w.qr + p1 / QTILE);
  MSC_LAUNCH_CHECK();
  group_ball_kernel<256, true><<<int(std::min(nk, most)), PR_T, 0, st>>>(X, d, dp, perm, nk, w.kc,
                                                                         w.kr);
  MSC_LAUNCH_CHECK();
  const int sgrid = int(std::max<int64_t>(1, std::min<int64_t>(ceil_div(ns, 8), num_sms() * 16)));
  sub_ball_kernel<<<sgrid, PR_T, 0, st>>>(X, d, dp, perm, leaf, zeros, ns, w.sc, w.sr, w.rsub);
  MSC_LAUNCH_CHECK();
  return MSC_OK;
}

int launch_nearest_tiles(const WorkItem* items, int64_t n_items, int d, const PruneWs& w,
                         int words, cudaStream_t st) {
  const int dp = int(round_up(d, 4));
  const int grid = int(std::max<int64_t>(1, std::min<int64_t>(ceil_div(n_items, 8),
                                                             int64_t(num_sms()) * 16)));
  nearest_tile_kernel<<<grid, PR_T, 0, st>>>(items, n_items, dp / 4, w.qc, w.kc, w.kr, words,
                                             w.mask);
  MSC_LAUNCH_CHECK();
  return MSC_OK;
}

int launch_query_plan(int d, const int32_t* perm, int64_t p1, int64_t n, int nb,
                      const WorkItem* items, int64_t n_items, const float* cand_thr,
                      const QStat* qs, const KeyMax* km, const Ctl* ctl, int prec, int kmma,
                      const PruneWs& w, int words, cudaStream_t st) {
  const int64_t nqblk = ceil_div(n, QTILE) * (QTILE / SUB);
  const int qgrid = int(std::max<int64_t>(1, std::min<int64_t>(ceil_div(nqblk * nb, 8),
                                                              int64_t(num_sms()) * 16)));
  query_radius_kernel<<<qgrid, PR_T, 0, st>>>(perm, p1, n, nb, cand_thr, qs, km, prec, kmma, d,
                                              nqblk, w.seed, w.rsub);
  MSC_LAUNCH_CHECK();
  const int dp = int(round_up(d, 4));
  const size_t smem = size_t(PLAN_WARPS) * 9 * dp * sizeof(float);
  int task_words;
  const int pgrid = plan_grid(n_items, words, task_words);
  // the plan indexes R by packed 32-row block: the queries' first block is p1 / 32
  plan_kernel<<<pgrid, PLAN_WARPS * 32, smem, st>>>(
      items, n_items, 256, d, dp, ctl, prec, w.qc, w.qr, w.kc, w.kr, w.sc, w.sr,
      w.rsub - p1 / SUB, words, w.mask, 0, PLAN_MAX_PAIRS, task_words, -1, nqblk);
  MSC_LAUNCH_CHECK();
  return MSC_OK;
}

PruneWs carve_query_prune(Carver& c, int64_t n, int64_t npk, int64_t p1, int d, int nb,
                          int64_t n_items, int words) {
  PruneWs w{};
  const int64_t npg = round_up(n, 256);
  w.leaf = c.take<int32_t>(npg);
  w.leaf2 = c.take<int32_t>(npk);
  w.perm2 = c.take<int32_t>(npg);
  w.reg = c.take<int32_t>(npg);
  w.S = c.take<int64_t>(npg + 1);
  w.scan_scratch = c.take<int64_t>(scan_i32_scratch_elems(npg));
  w.rpos = c.take<double>(std::max(npg, npk));
  w.mean = c.take<double>(1);
  w.mean_part = c.take<double2>(MEAN_CHUNKS);
  const int dp = int(round_up(d, 4));
  w.qc = c.take<float>(size_t(npk / QTILE + 1) * dp);
  w.qr = c.take<float>(npk / QTILE + 1);
  w.kc = c.take<float>(size_t(round_up(p1 / 256, 32)) * dp);
  w.kr = c.take<float>(p1 / 256);
  w.sc = c.take<float>(size_t(round_up(2 * npk / SUB, 32)) * dp);
  w.sr = c.take<float>(2 * npk / SUB);
  const int64_t nqblk = ceil_div(n, QTILE) * (QTILE / SUB);
  w.rsub = c.take<double>(std::max(npk / SUB, nqblk * nb));
  w.seed = c.take<float>(size_t(n) * nb);
  w.mask = c.take<uint32_t>(size_t(n_items) * words);
  w.vcnt = c.take<int32_t>(n_items);
  w.claim = c.take<int32_t>(n_items);
  w.chist = c.take<int32_t>(COST_BUCKETS);
  return w;
}

PruneWs carve_prune(Carver& c, int64_t npacked, int nseg, int d, int64_t n_items, int words,
                    int64_t n, int kprime) {
  PruneWs w{};
  w.leaf = c.take<int32_t>(npacked);
  w.leaf2 = c.take<int32_t>(npacked);
  w.perm2 = c.take<int32_t>(npacked);
  w.reg = c.take<int32_t>(npacked);
  w.S = c.take<int64_t>(npacked + 1);
  w.scan_scratch = c.take<int64_t>(scan_i32_scratch_elems(npacked));
  w.rpos = c.take<double>(npacked);
  w.rpos2 = c.take<double>(npacked);
  w.mean = c.take<double>(nseg);
  w.mean_part = c.take<double2>(size_t(nseg) * MEAN_CHUNKS);
  const int64_t nq = npacked / QTILE, nk = npacked / 256, ns = npacked / SUB;
  const int dp = int(round_up(d, 4));
  w.qc = c.take<float>(size_t(nq) * dp);
  w.qr = c.take<float>(nq);
  w.kc = c.take<float>(size_t(round_up(nk, 32)) * dp);          // interleaved in groups of 32
  w.kr = c.take<float>(nk);
  w.sc = c.take<float>(size_t(round_up(2 * ns, 32)) * dp);      // interleaved in groups of 32
  w.sr = c.take<float>(2 * ns);
  w.rsub = c.take<double>(ns);
  w.mask = c.take<uint32_t>(size_t(n_items) * words);
  w.mask3 = c.take<uint32_t>(size_t(n_items) * words);
  w.cand_val = c.take<float>(size_t(n) * kprime);
  w.iperm = c.take<int32_t>(n);
  w.excl = c.take<int4>(npacked);
  carve_refine_parts(c, w, int(std::min<int64_t>(256, n_items)), kprime);
  w.seed = c.take<float>(npacked);
  w.roff = c.take<double>(npacked);
  w.seed3 = c.take<float>(n);
  w.vcnt = c.take<int32_t>(n_items);
  w.claim = c.take<int32_t>(n_items);
  w.claim2 = c.take<int32_t>(n_items + int64_t(w.max_split_items) * (LONG_SPLIT - 1));
  w.chist = c.take<int32_t>(COST_BUCKETS);
  w.voff = c.take<int64_t>(n_items + 1);
  w.vscan = c.take<int64_t>(scan_i32_scratch_elems(n_items));
  // kept far tiles of all work items: at most every key tile of every work item; beyond a
  // quarter of that (pruning keeps a few percent on large samples) the mask walk takes over
  const int64_t all = n_items * int64_t(words) * 32;
  w.vcap = std::min<int64_t>(all, std::max<int64_t>(int64_t(16) << 20, all / 4));
  w.vlist = c.take<unsigned long long>(w.vcap);
  return w;
}

void carve_refine_parts(Carver& c, PruneWs& w, int max_items, int kprime) {
  w.max_split_items = max_items;
  const int64_t prow = int64_t(max_items) * REFINE_SPLIT * QTILE;
  w.part = c.take<int2>(size_t(prow) * kprime);
  w.part_thr = c.take<float>(prow);
}

int launch_prune_partition(const float* X, int d, const SegDesc* seg, int nseg, int64_t npacked,
                           int32_t* perm, const float* cand_thr, const QStat* qs,
                           const KeyMax* km, int prec, int kmma, int bn, const PruneWs& w,
                           cudaStream_t st) {
  (void)X;
  const int grid = grid_for(npacked);
  row_radius_kernel<<<grid, PR_T, 0, st>>>(perm, npacked, cand_thr, qs, km, prec, kmma, d, w.rpos);
  MSC_LAUNCH_CHECK();
  sample_mean_partial_kernel<<<dim3(MEAN_CHUNKS, std::min(nseg, 65535)), PR_T, 0, st>>>(
      seg, nseg, w.rpos, w.mean_part);
  MSC_LAUNCH_CHECK();
  sample_mean_final_kernel<<<(nseg + 127) / 128, 128, 0, st>>>(w.mean_part, nseg, w.mean);
  MSC_LAUNCH_CHECK();
  double factor = OUTLIER_FACTOR;
  if (const char* env = std::getenv("MSC_B200_OUTLIER_FACTOR")) {
    const double v = std::atof(env);
    if (v > 1.0) factor = v;
  }
  regular_flag_kernel<<<grid, PR_T, 0, st>>>(perm, npacked, seg, nseg, w.rpos, w.mean, factor,
                                             w.reg);
  MSC_LAUNCH_CHECK();
  MSC_TRY(scan_excl_i32(w.reg, npacked, w.S, w.scan_scratch, st));
  partition_kernel<<<grid, PR_T, 0, st>>>(perm, w.leaf, w.rpos, npacked, seg, nseg, w.reg, w.S,
                                          cand_thr, qs, km, prec, kmma, d, bn, w.perm2,
                                          w.leaf2, w.rpos2, w.seed, w.iperm, w.excl);
  MSC_LAUNCH_CHECK();
  MSC_CUDA_TRY(cudaMemcpyAsync(perm, w.perm2, sizeof(int32_t) * npacked,
                               cudaMemcpyDeviceToDevice, st));
  return MSC_OK;
}

int prune_counters(unsigned long long* out) {
  MSC_CUDA_TRY(cudaMemcpyFromSymbol(out, g_prune_tiles, sizeof(unsigned long long) * 6));
  return MSC_OK;
}
int prune_counters_clear() {
  const unsigned long long z[6] = {};
  MSC_CUDA_TRY(cudaMemcpyToSymbol(g_prune_tiles, z, sizeof(z)));
  return MSC_OK;
}

int launch_prune_plan(const float* X, int d, int64_t npacked, const int32_t* perm,
                      const WorkItem* items, int64_t n_items, int bn, const Ctl* ctl, int prec,
                      const PruneWs& w, int words, cudaStream_t st) {
  if (d > 128 || bn > 256 || (npacked % 256) != 0) {
    set_error("prune plan: unsupported shape (d=%d, bn=%d)", d, bn);
    return MSC_ERR_INVALID_ARG;
  }
  const int64_t nq = npacked / QTILE, nk = npacked / 256, ns = npacked / SUB;
  const int dp = int(round_up(d, 4));
  const int64_t most = int64_t(num_sms()) * 32;
  group_ball_kernel<QTILE, false><<<int(std::min(nq, most)), PR_T, 0, st>>>(X, d, dp, perm, nq,
                                                                           w.qc, w.qr);
  MSC_LAUNCH_CHECK();
  group_ball_kernel<256, true><<<int(std::min(nk, most)), PR_T, 0, st>>>(X, d, dp, perm, nk, w.kc,
                                                                         w.kr);
  MSC_LAUNCH_CHECK();
  const int sgrid = int(std::max<int64_t>(1, std::min<int64_t>(ceil_div(ns, 8), num_sms() * 16)));
  sub_ball_kernel<<<sgrid, PR_T, 0, st>>>(X, d, dp, perm, w.leaf2, w.rpos2, ns, w.sc, w.sr, w.rsub);
  MSC_LAUNCH_CHECK();
  const size_t smem = size_t(PLAN_WARPS) * 9 * dp * sizeof(float);
  int max_pairs = PLAN_MAX_PAIRS;
  if (const char* env = std::getenv("MSC_B200_PLAN_PAIRS")) max_pairs = std::max(0, std::atoi(env));
  int task_words;
  const int pgrid = plan_grid(n_items, words, task_words);
  plan_kernel<<<pgrid, PLAN_WARPS * 32, smem, st>>>(items, n_items, bn, d, dp, ctl, prec, w.qc,
                                                    w.qr, w.kc, w.kr, w.sc, w.sr, w.rsub, words,
                                                    w.mask, profiling_enabled() ? 1 : 0,
                                                    max_pairs, task_words, 2, 0);
  MSC_LAUNCH_CHECK();
  // point test of the kept pairs, opt-in (MSC_B200_POINT_TEST=1).  Measured at 1.3M × 50: far
  // tiles kept 2.63 M → 1.63 M and main scan 33.4 → 28.0 ms, but the test itself costs ~15 ms
  // (every key of a separated pair is checked over all d dimensions on the CUDA cores), so the
  // graph takes 81.0 ms against 72.6 without it
  const char* pt_env = std::getenv("MSC_B200_POINT_TEST");
  if ((pt_env && *pt_env == '1') && bn == 256) {
    const size_t psmem = size_t(256) * d * sizeof(float);
    MSC_CUDA_TRY(raise_smem_cap(point_test_kernel, psmem));
    const int64_t nblk = nk * POINT_SLICES;
    const int ptgrid = int(std::max<int64_t>(1, std::min<int64_t>(nblk, int64_t(num_sms()) * 8)));
    point_test_kernel<<<ptgrid, POINT_T, psmem, st>>>(X, d, dp, perm, items, n_items, bn, words,
                                                      ctl, prec, w.qc, w.qr, w.rsub, w.mask, nk,
                                                      profiling_enabled() ? 1 : 0);
    MSC_LAUNCH_CHECK();
  }
  return MSC_OK;
}

int launch_claim_order(int64_t n_items, int words, const PruneWs& w, cudaStream_t st) {
  const int cgrid = int(std::max<int64_t>(1, std::min<int64_t>(ceil_div(n_items, 8),
                                                              int64_t(num_sms()) * 8)));
  visit_count_kernel<<<cgrid, PR_T, 0, st>>>(w.mask, n_items, words, w.vcnt);
  MSC_LAUNCH_CHECK();
  int shift = 0;
  while ((int64_t(words) * 32 >> shift) >= COST_BUCKETS) ++shift;
  MSC_CUDA_TRY(cudaMemsetAsync(w.chist, 0, sizeof(int32_t) * COST_BUCKETS, st));
  const int hgrid = int(std::max<int64_t>(1, std::min<int64_t>(ceil_div(n_items, PR_T),
                                                              int64_t(num_sms()) * 2)));
  cost_hist_kernel<<<hgrid, PR_T, 0, st>>>(w.vcnt, n_items, shift, w.chist);
  MSC_LAUNCH_CHECK();
  cost_offsets_kernel<<<1, COST_BUCKETS, 0, st>>>(w.chist);
  MSC_LAUNCH_CHECK();
  cost_scatter_kernel<<<hgrid, PR_T, 0, st>>>(w.vcnt, n_items, shift, w.chist, w.claim);
  MSC_LAUNCH_CHECK();
  return MSC_OK;
}

int launch_refine_seed(const int32_t* qmap, const int32_t* n_rows, int64_t max_rows,
                       const int32_t* perm, const float* cand_thr, const QStat* qs,
                       const KeyMax* km, const QStat* qs3, const KeyMax* km3, const Ctl* ctl,
                       int prec, int kmma, int kmma3, int d, const PruneWs& w, cudaStream_t st) {
  refine_seed_kernel<<<grid_for(max_rows), PR_T, 0, st>>>(qmap, n_rows, perm, cand_thr, w.seed,
                                                          w.excl, qs, km, qs3, km3, ctl, prec,
                                                          kmma, kmma3, d, w.seed3);
  MSC_LAUNCH_CHECK();
  return MSC_OK;
}

int launch_long_plan(int64_t n_items, int words, int n_ctas, const PruneWs& w, Ctl* ctl,
                     cudaStream_t st) {
  int shift = 0;
  while ((int64_t(words) * 32 >> shift) >= COST_BUCKETS) ++shift;
  long_plan_kernel<<<1, LONG_T, 0, st>>>(w.vcnt, n_items, shift, n_ctas, w.max_split_items,
                                         w.claim, w.claim2, ctl, profiling_enabled() ? 1 : 0);
  MSC_LAUNCH_CHECK();
  return MSC_OK;
}

int launch_long_merge(const WorkItem* items, const Ctl* ctl, const int32_t* perm,
                      const PruneWs& w, int kprime, int kper, int32_t* cand_idx,
                      float* cand_thr, cudaStream_t st) {
  const int grid = int(std::max<int64_t>(
      1, std::min<int64_t>(int64_t(w.max_split_items) * QTILE / 8, int64_t(num_sms()) * 8)));
  long_merge_kernel<<<grid, PR_T, 0, st>>>(items, ctl, w.claim, perm, w.part, w.part_thr,
                                           w.cand_val, kprime, kper, cand_idx, cand_thr, w.seed,
                                           w.excl);
  MSC_LAUNCH_CHECK();
  return MSC_OK;
}

int launch_visit_order(const WorkItem* items, int64_t n_items, int bn, int d, int64_t npacked,
                       const int32_t* perm, const Ctl* ctl, Ctl* ctl_w, int prec, int kmma,
                       const QStat* qs, const KeyMax* km, const PruneWs& w, int words,
                       cudaStream_t st, bool* built) {
  *built = false;
  // opt-in (MSC_B200_ORDERED=1): on clustered 50-dimensional data the nearest-ball-first order
  // left the insertions per row and the scanned tiles almost unchanged (the rows of one cluster
  // are nearly equidistant), and building the lists cost about what the main scan saved
  const char* env = std::getenv("MSC_B200_ORDERED");
  if (!(env && *env == '1')) return MSC_OK;
  const int dp = int(round_up(d, 4));
  const size_t smem = size_t(VO_SORT_MAX) * 16 + size_t(dp) * 4 + size_t(words + 1) * 4;
  if (bn != 256 || d > 128 || smem > size_t(200) * 1024) return MSC_OK;
  row_offset_kernel<<<grid_for(npacked), PR_T, 0, st>>>(perm, npacked, qs, km, prec, kmma, d,
                                                        w.roff);
  MSC_LAUNCH_CHECK();
  const int cgrid = int(std::max<int64_t>(1, std::min<int64_t>(ceil_div(n_items, 8),
                                                              int64_t(num_sms()) * 8)));
  visit_count_kernel<<<cgrid, PR_T, 0, st>>>(w.mask, n_items, words, w.vcnt);
  MSC_LAUNCH_CHECK();
  MSC_TRY(scan_excl_i32(w.vcnt, n_items, w.voff, w.vscan, st));
  MSC_CUDA_TRY(raise_smem_cap(visit_order_kernel, smem));
  const int ogrid = int(std::max<int64_t>(1, std::min<int64_t>(n_items, int64_t(num_sms()) * 4)));
  visit_order_kernel<<<ogrid, VO_T, smem, st>>>(items, n_items, bn, d, dp, ctl, prec, w.qc, w.qr,
                                                w.kc, w.kr, w.mask, words, w.voff, w.vcap,
                                                w.vlist, &ctl_w->ordered_ok);
  MSC_LAUNCH_CHECK();
  *built = true;
  return MSC_OK;
}

int launch_refine_mask(const WorkItem* items3, const int32_t* n_items3, const int32_t* qmap,
                       int64_t max_items, const SegDesc* seg, int nseg, int bn, int words,
                       const QStat* qs, const KeyMax* km, const QStat* qs3, const KeyMax* km3,
                       const Ctl* ctl, int prec, int kmma, int kmma3, int d, const PruneWs& w,
                       cudaStream_t st) {
  const int grid = int(std::max<int64_t>(1, std::min<int64_t>(ceil_div(max_items, 8),
                                                             int64_t(num_sms()) * 8)));
  refine_mask_kernel<<<grid, PR_T, 0, st>>>(items3, n_items3, qmap, seg, nseg, w.mask, words, bn,
                                            qs, km, qs3, km3, ctl, prec, kmma, kmma3, d, w.mask3);
  MSC_LAUNCH_CHECK();
  return MSC_OK;
}

int launch_refine_merge(const WorkItem* items3, const int32_t* n_items3, const Ctl* ctl,
                        const int32_t* qmap, const int32_t* perm, int64_t max_rows,
                        const PruneWs& w, int kprime, int32_t* cand_idx, float* cand_thr,
                        cudaStream_t st) {
  const int64_t rows = std::min<int64_t>(max_rows, int64_t(w.max_split_items) * QTILE);
  const int grid = int(std::max<int64_t>(1, std::min<int64_t>(ceil_div(rows, 8),
                                                             int64_t(num_sms()) * 8)));
  refine_merge_kernel<<<grid, PR_T, 0, st>>>(items3, n_items3, ctl, qmap, perm, w.part,
                                             w.part_thr, kprime, cand_idx, cand_thr);
  MSC_LAUNCH_CHECK();
  return MSC_OK;
}

}  // namespace msc
