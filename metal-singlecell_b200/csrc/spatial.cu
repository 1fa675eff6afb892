// Uniform-grid (cell-list) exact kNN and fixed-radius search of 2-D / 3-D coordinates: the
// spatial index of metalsinglecell's neighbors._knn_grid / _radius_grid (neighbors.py:143-417),
// which gr.spatial_neighbors_knn / _radius (gr.py:186-255) and spatial.spatial_neighbors
// (spatial.py:13-44) call.
//
// Arithmetic (the reference grid kernel's, neighbors.py:180-183, fixed so that every row follows
// it): d² = fl(fl(dx²) + fl(dy²)) [+ fl(dz²)], dx = fl(x_p − x_q), no fused multiply-add;
// distance = correctly rounded float32 sqrt(d²); kNN order (distance, index) with self first;
// radius test r_lo² ≤ d² ≤ r_hi² with r² rounded once to float32 (neighbors.py:301-302).
//
// Build, all on the device:
//   sp_bbox   per-axis minimum / maximum (order-preserving integer atomics), non-finite count
//   sp_plan   one thread: cell side, cells per axis (at most 4n + 16 cells), FP64 geometry
//   sp_bin    cell of every point (FP64 floor of (x − o) / cs), cell counts
//   scan      cell starts
//   sp_place  points in cell order as float4 (x, y, z, index bits)
// Search: one lane per query, the queries in cell order, each lane walking its own cells.  Lanes of
// one cell read the same points at the same time and lanes of neighbouring cells nearly the same
// lines.  (A warp per cell with the candidates staged for all its lanes left most lanes without a
// query where cells hold few points, and so wanted large cells, whose candidates are mostly too
// far.  1M spots, k = 7, whole search: 1.86 ms, now 0.55.)
//   kNN: the 3^d cells around the query's cell, then larger boxes; a lane keeps its k − 1
//        best (distance, index) keys sorted in registers; it is done once its (k−1)-th distance
//        is provably below the distance to every cell outside the scanned box (FP64 bound with a
//        margin that covers float32 rounding), so every row is exact without a fallback pass.
//   radius: every cell within ring = ceil(D / cs) of the query's cell, D = radius plus a margin
//        that covers rounding; a count pass, a scan, a fill pass in the same walk order, then
//        each row's columns put in ascending order (rank sort).
#include <climits>

#include "kernels.cuh"

namespace msc {

namespace {

constexpr int SP_T = 128;                 // threads per block of the search kernels
constexpr int SP_W = SP_T / 32;
constexpr int LANE_R = 4;                 // kNN: largest box of cells one lane walks
constexpr int LANE_UNROLL_K = 16;         // ... longest list whose insertion is worth copying
constexpr int FAR_FIRST = 8;              // ... points of it in the first pass / list length
constexpr int FAR_RUN = 32;               // ... most points of a row of cells it reads alone
constexpr double CELL_PER_K = 0.33;       // kNN in the plane: points per cell / k
constexpr int SORT_TILE = 256;            // columns staged per warp by the row sort
constexpr int SORT_E = 4;                 // entries ranked per lane per group

struct SpGrid {
  double o[3];          // origin (per-axis minimum)
  double cs;            // cell side
  double eps_abs;       // absolute slack of FP64 geometry
  double reach;         // radius search: D
  int32_t g[3];         // cells per axis (1 on an unused axis)
  int32_t ring;         // radius search: cells scanned on each side
  int64_t ncells;
  int32_t status;       // 0 ok, 1 non-finite coordinates, 2 plan failed
  int32_t pad;
};

__device__ __forceinline__ int64_t imin64(int64_t a, int64_t b) { return a < b ? a : b; }

__device__ __forceinline__ unsigned f2o(float f) {
  unsigned u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float o2f(unsigned u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// mm[0..2] = ordered minima, mm[3..5] = ordered maxima (initialised to 0xffffffff / 0)
__global__ void sp_bbox_kernel(const float* __restrict__ X, int64_t n, int d,
                               unsigned* __restrict__ mm, unsigned long long* __restrict__ nonfinite) {
  float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  unsigned long long bad = 0;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    for (int a = 0; a < d; ++a) {
      float v = X[i * d + a];
      if (!isfinite(v)) { ++bad; continue; }
      lo[a] = fminf(lo[a], v);
      hi[a] = fmaxf(hi[a], v);
    }
  }
  for (int a = 0; a < d; ++a) {
    for (int off = 16; off > 0; off >>= 1) {
      lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], off));
      hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], off));
    }
  }
  for (int off = 16; off > 0; off >>= 1) bad += __shfl_xor_sync(0xffffffffu, bad, off);
  // one set of atomics per block (one per warp took 53 us at 1M points)
  __shared__ float slo[3][32], shi[3][32];
  __shared__ unsigned long long sbad[32];
  const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    for (int a = 0; a < 3; ++a) { slo[a][w] = lo[a]; shi[a][w] = hi[a]; }
    sbad[w] = bad;
  }
  __syncthreads();
  if (threadIdx.x < d) {
    const int a = threadIdx.x;
    float l = slo[a][0], h = shi[a][0];
    for (int i = 1; i < nw; ++i) { l = fminf(l, slo[a][i]); h = fmaxf(h, shi[a][i]); }
    if (l <= h) {
      atomicMin(&mm[a], f2o(l));
      atomicMax(&mm[3 + a], f2o(h));
    }
  }
  if (threadIdx.x == 0) {
    for (int i = 1; i < nw; ++i) bad += sbad[i];
    if (bad) atomicAdd(nonfinite, bad);
  }
}

// mode 0: kNN (k), mode 1: radius (reach = D > 0)
__global__ void sp_plan_kernel(const unsigned* __restrict__ mm,
                               const unsigned long long* __restrict__ nonfinite, int64_t n, int d,
                               int mode, int k, double reach, SpGrid* __restrict__ G) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  SpGrid g{};
  g.reach = reach;
  if (*nonfinite) { g.status = 1; *G = g; return; }
  double ext[3] = {0, 0, 0};
  double mag = 0;
  int eff = 0;
  for (int a = 0; a < 3; ++a) {
    if (a < d) {
      const double lo = double(o2f(mm[a])), hi = double(o2f(mm[3 + a]));
      g.o[a] = lo;
      ext[a] = hi - lo;
      mag = fmax(mag, fmax(fabs(lo), fabs(hi)));
      if (ext[a] > 0) ++eff;
    } else {
      g.o[a] = 0;
    }
  }
  double cs;
  if (mode == 0) {
    if (eff == 0) {
      cs = 1.0;
    } else {
      // points per cell on average: of the 3^d cells scanned first a circle (ball) of one cell
      // side around the query is certain to be covered, so about k/3 points a cell in the plane and
      // k/4 in space end most walks there where the points are as dense as on average; in denser
      // regions, where most points are, cells hold more.  (1M spots of uneven density, k = 7: whole
      // search 0.67 ms at 0.33 k points a cell, 0.79 at 0.5 k.)
      // Where an axis spans few cells the points lie as along a line (or in a plane), of which a
      // box covers less: the side is the largest of those that the one, two and three longest axes
      // ask for.  (2,094 points along a line, k = 45, as cells of a plane: 1.08 ms, every query
      // beyond its first box; now 0.41.)
      double e[3] = {ext[0], ext[1], ext[2]};                     // descending
      if (e[0] < e[1]) { const double t = e[0]; e[0] = e[1]; e[1] = t; }
      if (e[1] < e[2]) { const double t = e[1]; e[1] = e[2]; e[2] = t; }
      if (e[0] < e[1]) { const double t = e[0]; e[0] = e[1]; e[1] = t; }
      const double per[3] = {0.7 * k, CELL_PER_K * k, 0.25 * k};  // points per cell
      double vol = 1.0;
      cs = 0.0;
      for (int a = 0; a < eff; ++a) {
        vol *= e[a];
        cs = fmax(cs, pow(fmax(1.0, per[a]) * vol / double(n), 1.0 / (a + 1)));
      }
    }
  } else {
    cs = reach > 0 ? reach * (1.0 + 1e-6) : 1.0;
  }
  const double cap = 4.0 * double(n) + 16.0;
  double cells = 0;
  bool ok = false;
  for (int it = 0; it < 200; ++it) {
    cells = 1;
    for (int a = 0; a < 3; ++a) cells *= ext[a] > 0 ? ceil(ext[a] / cs) + 1.0 : 1.0;
    if (cells <= cap) { ok = true; break; }
    if (!isfinite(cells) || !(cs > 0)) {
      // a cell side so small that the cell count overflows: restart from two cells per axis
      cs = fmax(fmax(ext[0], ext[1]), ext[2]) * 0.5;
      continue;
    }
    cs *= pow(cells / cap, 1.0 / (eff > 0 ? eff : 1)) * (1.0 + 1e-9);
  }
  if (!ok || !(cs > 0) || !isfinite(cs)) { g.status = 2; *G = g; return; }
  for (int a = 0; a < 3; ++a) g.g[a] = ext[a] > 0 ? int32_t(ceil(ext[a] / cs) + 1.0) : 1;
  g.ncells = int64_t(g.g[0]) * g.g[1] * g.g[2];
  g.cs = cs;
  g.eps_abs = 1e-12 * (mag + cs);
  if (mode == 1) {
    const double r = reach / cs + 1e-7;
    int ring = int(ceil(r));
    int gmax = max(g.g[0], max(g.g[1], g.g[2]));
    g.ring = max(1, min(ring, gmax));
  }
  *G = g;
}

__device__ __forceinline__ int cell_axis(float x, const SpGrid& g, int a) {
  const double t = floor((double(x) - g.o[a]) / g.cs);
  int c = t < 0 ? 0 : (t > double(g.g[a] - 1) ? g.g[a] - 1 : int(t));
  return c;
}

__device__ __forceinline__ int64_t cell_of(const float* p, int d, const SpGrid& g) {
  const int cx = cell_axis(p[0], g, 0);
  const int cy = cell_axis(p[1], g, 1);
  const int cz = d == 3 ? cell_axis(p[2], g, 2) : 0;
  return (int64_t(cz) * g.g[1] + cy) * g.g[0] + cx;
}

__global__ void sp_bin_kernel(const float* __restrict__ X, int64_t n, int d,
                              const SpGrid* __restrict__ G, int64_t* __restrict__ cell,
                              int32_t* __restrict__ count) {
  const SpGrid g = *G;
  if (g.status) return;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t c = cell_of(X + i * d, d, g);
    cell[i] = c;
    atomicAdd(&count[c], 1);
  }
}

__global__ void sp_place_kernel(const float* __restrict__ X, int64_t n, int d,
                                const SpGrid* __restrict__ G, const int64_t* __restrict__ cell,
                                const int64_t* __restrict__ cell_start, int32_t* __restrict__ cursor,
                                float4* __restrict__ pts) {
  if (G->status) return;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t c = cell[i];
    const int64_t pos = cell_start[c] + atomicAdd(&cursor[c], 1);
    const float* p = X + i * d;
    pts[pos] = make_float4(p[0], p[1], d == 3 ? p[2] : 0.f, __int_as_float(int(i)));
  }
}

template <int D>
__device__ __forceinline__ float sq_dist(const float4& p, const float4& q) {
  const float dx = __fsub_rn(p.x, q.x);
  float s = __fmul_rn(dx, dx);
  const float dy = __fsub_rn(p.y, q.y);
  s = __fadd_rn(s, __fmul_rn(dy, dy));
  if (D == 3) {
    const float dz = __fsub_rn(p.z, q.z);
    s = __fadd_rn(s, __fmul_rn(dz, dz));
  }
  return s;
}

__device__ __forceinline__ bool key_less(float s, int i, float ts, int ti) {
  return s < ts || (s == ts && i < ti);
}

// d² above this cannot give a distance ≤ top: (next float above top)², rounded up
__device__ __forceinline__ float prefilter(float top) {
  if (top < 0.f) return -1.f;
  if (isinf(top)) return INFINITY;
  const float up = __uint_as_float(__float_as_uint(top) + 1u);
  return __fmul_ru(up, up);
}

// f(point) for the points [a, b), four loads in flight
template <class F>
__device__ __forceinline__ void scan_run(const float4* __restrict__ pts, int64_t a, int64_t b,
                                         F&& f) {
  for (; a + 4 <= b; a += 4) {
    const float4 p0 = pts[a], p1 = pts[a + 1], p2 = pts[a + 2], p3 = pts[a + 3];
    f(p0);
    f(p1);
    f(p2);
    f(p3);
  }
  for (; a < b; ++a) f(pts[a]);
}

// hit(d2, id) for those of `len` points whose squared distance to q passes test(d2), few of them.
// Four points at a time: their loads and distances do not wait for one another, and one branch
// passes over all four.
template <int D, class T, class F>
__device__ __forceinline__ void scan_hits(const float4* __restrict__ at, int len, const float4& q,
                                          T&& test, F&& hit) {
  int t = 0;
  for (; t + 4 <= len; t += 4) {
    float d2[4];
    int id[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float4 p = at[t + u];
      d2[u] = sq_dist<D>(p, q);
      id[u] = __float_as_int(p.w);
    }
    if (test(fminf(fminf(d2[0], d2[1]), fminf(d2[2], d2[3])))) {
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (test(d2[u])) hit(d2[u], id[u]);
    }
  }
  for (; t < len; ++t) {
    const float4 p = at[t];
    const float d2 = sq_dist<D>(p, q);
    if (test(d2)) hit(d2, __float_as_int(p.w));
  }
}

// blocks per SM by list length: latency-bound walks want warps (K = 8: 0.67 -> 0.55 ms at 10
// blocks), long lists registers (K = 32: 42,319 points in space 14.5 -> 10.9 ms at 3 for 4).  0: no
// bound, the compiler's choice (K = 64: 168 registers; uniform 100,000, k = 65, 1.5 ms, 2.0 at 2)
constexpr int knn_blocks(int K) { return K <= 8 ? 10 : (K <= 16 ? 6 : (K <= 32 ? 3 : 0)); }
template <int K, int D>
__global__ void __launch_bounds__(SP_T, knn_blocks(K))
sp_knn_kernel(const float4* __restrict__ pts, const int64_t* __restrict__ cell_start,
              const SpGrid* __restrict__ G, int64_t n, int k, int32_t* __restrict__ out_idx,
              float* __restrict__ out_dist, unsigned long long* __restrict__ counters,
              int32_t* __restrict__ far_rows, int32_t* __restrict__ n_far) {
  const SpGrid g = *G;
  if (g.status) return;
  const int lane = threadIdx.x & 31;
  const int m = k - 1;
  unsigned long long evals = 0, expanded = 0;
  for (int64_t pos = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; pos < n;
       pos += int64_t(gridDim.x) * blockDim.x) {
    const float4 q = pts[pos];
    const int qi = __float_as_int(q.w);
    const int cx = cell_axis(q.x, g, 0), cy = cell_axis(q.y, g, 1);
    const int cz = D == 3 ? cell_axis(q.z, g, 2) : 0;
    float s[K];
    int id[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const bool sent = j < K - m;
      s[j] = sent ? -1.f : INFINITY;
      id[j] = sent ? -1 : INT_MAX;
    }
    float t2 = prefilter(s[K - 1]);
    const int rmax = max(max(cx, g.g[0] - 1 - cx),
                         max(max(cy, g.g[1] - 1 - cy), D == 3 ? max(cz, g.g[2] - 1 - cz) : 0));
    auto insert = [&](float d2, int pid) {
      const float sd = __fsqrt_rn(d2);
      if (pid == qi || !key_less(sd, pid, s[K - 1], id[K - 1])) return;
#pragma unroll
      for (int j = K - 1; j > 0; --j) {
        const bool lp = key_less(sd, pid, s[j - 1], id[j - 1]);
        const bool lc = key_less(sd, pid, s[j], id[j]);
        const float ns = lp ? s[j - 1] : (lc ? sd : s[j]);
        const int ni = lp ? id[j - 1] : (lc ? pid : id[j]);
        s[j] = ns;
        id[j] = ni;
      }
      if (key_less(sd, pid, s[0], id[0])) { s[0] = sd; id[0] = pid; }
      t2 = prefilter(s[K - 1]);
    };
    // The points of cells x0..x1 of a row of cells, four at a time.  The insertion is K steps of code,
    // some 8 KB at K = 64: copied for every point and every place that scans a run it did not stay in
    // the instruction cache.  So there is one such place, and lists beyond LANE_UNROLL_K insert a
    // group's hits in a loop: uniform 100,000 points, k = 65, 3.6 -> 2.0 ms, in space 7.8 -> 3.3; a
    // slide of uneven density, 274,473 spots, k = 40, 121 -> 47.  The unrolled groups serve the short
    // lists better (1M spots, k = 7: 0.52 against 0.67 ms).
    auto run = [&](int y, int z, int x0, int x1) {
      x0 = max(x0, 0);
      x1 = min(x1, g.g[0] - 1);
      if (x0 > x1) return;
      const int64_t row = (int64_t(z) * g.g[1] + y) * g.g[0];
      const int64_t a = cell_start[row + x0];
      const int len = int(cell_start[row + x1 + 1] - a);
      const float4* at = pts + a;
      evals += len;
      if constexpr (K <= LANE_UNROLL_K) {
        scan_hits<D>(at, len, q, [&](float d2) { return d2 <= t2; }, insert);
        return;
      }
#pragma unroll 1
      for (int t = 0; t < len; t += 4) {
        float d2[4];
        int pid[4];
        unsigned m = 0u;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float4 p = at[min(t + u, len - 1)];
          d2[u] = sq_dist<D>(p, q);
          pid[u] = __float_as_int(p.w);
          if (d2[u] <= t2 && t + u < len) m |= 1u << u;
        }
#pragma unroll 1
        for (; m; m &= m - 1) {
          const bool odd = (m & 0xAu & (0u - m)) != 0u, high = (m & 3u) == 0u;
          insert(high ? (odd ? d2[3] : d2[2]) : (odd ? d2[1] : d2[0]),
                 high ? (odd ? pid[3] : pid[2]) : (odd ? pid[1] : pid[0]));
        }
      }
    };
    // Boxes of cells |d| <= R around the query's cell, R = 1 first; the cells of the last box (P) are
    // left out of the next, and rows of cells beyond the list's last distance r are skipped.  r says
    // which box is enough; a query that is not done within LANE_R (far from other points) goes to
    // the warp pass: its one lane would walk thousands of row ranges while the launch waits.
    bool defer = false;
    for (int P = -1, R = 1;;) {
      // the query's own row of cells first (its near points bound the list early: 1M spots, k = 7,
      // 0.57 -> 0.52 ms), then outwards: 0, -1, 1, -2, ...
      for (int tz = 0; tz <= (D == 3 ? 2 * R : 0); ++tz) {
        const int dz = (tz & 1) ? -((tz + 1) >> 1) : tz >> 1;
        if (D == 3 && (cz + dz < 0 || cz + dz >= g.g[2])) continue;
#pragma unroll 1
        for (int ty = 0; ty <= 2 * R; ++ty) {
          const int dy = (ty & 1) ? -((ty + 1) >> 1) : ty >> 1;
          if (cy + dy < 0 || cy + dy >= g.g[1]) continue;
          if (P >= 1) {
            const double far = double(s[K - 1]) * (1.0 + 4e-6) + g.eps_abs;
            const double ly = g.o[1] + double(cy + dy) * g.cs;           // the row's lower face
            if (ly - double(q.y) > far || double(q.y) - (ly + g.cs) > far) continue;
            if (D == 3) {
              const double lz = g.o[2] + double(cz + dz) * g.cs;
              if (lz - double(q.z) > far || double(q.z) - (lz + g.cs) > far) continue;
            }
          }
          // all of the row, or its cells on either side of the last box
          const bool full = abs(dy) > P || (D == 3 && abs(dz) > P);
#pragma unroll 1
          for (int side = full ? 1 : 0; side < 2; ++side)
            run(cy + dy, cz + dz, full || side == 0 ? cx - R : cx + P + 1,
                full || side == 1 ? cx + R : cx - P - 1);
        }
      }
      // distance from the query to the nearest face of the box of cells within R that has
      // points beyond it; a box that reaches the grid's edge on a side bounds nothing there
      double bound = INFINITY;
      const int cc[3] = {cx, cy, cz};
      const float qq[3] = {q.x, q.y, q.z};
#pragma unroll
      for (int a = 0; a < D; ++a) {
        if (cc[a] - R > 0)
          bound = fmin(bound, double(qq[a]) - (g.o[a] + double(cc[a] - R) * g.cs));
        if (cc[a] + R < g.g[a] - 1)
          bound = fmin(bound, (g.o[a] + double(cc[a] + R + 1) * g.cs) - double(qq[a]));
      }
      const double r = double(s[K - 1]);
      if (isinf(bound) || r < bound * (1.0 - 4e-6) - g.eps_abs || R >= rmax) {
        if (R >= 2) ++expanded;
        break;
      }
      P = R;
      // the faces of box R lie at least R·cs away, so R > r / cs ends the walk
      const double want = isinf(r) ? double(R + 1) : r * (1.0 + 1e-5) / g.cs + 1.0;
      R = max(R + 1, int(fmin(want, double(rmax))));
      if (R > LANE_R) { defer = true; break; }
    }
    if (defer) {
      far_rows[atomicAdd(n_far, 1)] = int32_t(pos);
      ++expanded;
      continue;
    }
    int32_t* oi = out_idx + int64_t(qi) * k;
    float* od = out_dist + int64_t(qi) * k;
    oi[0] = qi;
    od[0] = 0.f;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      if (j >= K - m) {
        oi[1 + j - (K - m)] = id[j];
        od[1 + j - (K - m)] = s[j];
      }
    }
  }
  __syncwarp();
  for (int off = 16; off > 0; off >>= 1) {
    evals += __shfl_xor_sync(0xffffffffu, evals, off);
    expanded += __shfl_xor_sync(0xffffffffu, expanded, off);
  }
  if (lane == 0) {
    atomicAdd(&counters[0], evals);
    atomicAdd(&counters[1], expanded);
  }
}

// The queries the lane pass left open, a warp each: the lanes share a box's rows of cells.  First the
// smallest box of a doubling sequence that holds k points (from the cell starts alone), then that
// box's (k-1)-th distance r, then the rows and cells within r: every point that can be nearer.
// Each lane keeps a sorted list of what it sees; the warp takes the smallest head m times.  Any k
// points bound the distance, so the first pass takes only a few of a long row: 46,931 points with
// three far outliers 7.1 -> 6.4 ms.
template <int K, int D>
__global__ void __launch_bounds__(SP_T)
sp_knn_far_kernel(const float4* __restrict__ pts, const int64_t* __restrict__ cell_start,
                  const SpGrid* __restrict__ G, int k, const int32_t* __restrict__ far_rows,
                  const int32_t* __restrict__ n_far, int32_t* __restrict__ out_idx,
                  float* __restrict__ out_dist, unsigned long long* __restrict__ counters) {
  const SpGrid g = *G;
  if (g.status) return;
  const int lane = threadIdx.x & 31;
  const int m = k - 1, total = *n_far;
  unsigned long long evals = 0;
  for (int w = int((blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5); w < total;
       w += int((int64_t(gridDim.x) * blockDim.x) >> 5)) {
    const float4 q = pts[far_rows[w]];
    const int qi = __float_as_int(q.w);
    const int c[3] = {cell_axis(q.x, g, 0), cell_axis(q.y, g, 1),
                      D == 3 ? cell_axis(q.z, g, 2) : 0};
    const float qq[3] = {q.x, q.y, q.z};
    int rmax = 0;
#pragma unroll
    for (int a = 0; a < D; ++a) rmax = max(rmax, max(c[a], g.g[a] - 1 - c[a]));
    // f(first, step, last + 1) for the points of box R, cut to the cells within r: a lane takes a
    // row of cells, and a row of more than FAR_RUN points goes to the whole warp (a lone lane
    // reading the 30,000 points of one cell is a load latency for each: 11 ms).
    auto rows = [&](int R, double r, auto&& f) {
      const int y0 = max(c[1] - R, 0), y1 = min(c[1] + R, g.g[1] - 1), ny = y1 - y0 + 1;
      const int z0 = D == 3 ? max(c[2] - R, 0) : 0, z1 = D == 3 ? min(c[2] + R, g.g[2] - 1) : 0;
      const int64_t nrow = int64_t(ny) * (z1 - z0 + 1);
      for (int64_t e0 = 0; e0 < nrow; e0 += 32) {  // warp-uniform
        const int64_t e = e0 + lane;
        int64_t a = 0, b = 0;
        if (e < nrow) {
          const int y = y0 + int(e % ny), z = z0 + int(e / ny);
          double rest = r * r;                     // (reach along x)², from the row's distance
          const double ly = g.o[1] + double(y) * g.cs;
          const double ey = fmax(0.0, fmax(ly - double(qq[1]), double(qq[1]) - (ly + g.cs)));
          rest -= ey * ey;
          if (D == 3) {
            const double lz = g.o[2] + double(z) * g.cs;
            const double ez = fmax(0.0, fmax(lz - double(qq[2]), double(qq[2]) - (lz + g.cs)));
            rest -= ez * ez;
          }
          int x0 = max(c[0] - R, 0), x1 = min(c[0] + R, g.g[0] - 1);
          if (rest < 1e300) {                      // one cell to spare on either side
            const double h = sqrt(fmax(rest, 0.0)) / g.cs + 1.0;
            const double at = (double(qq[0]) - g.o[0]) / g.cs;
            x0 = max(x0, int(fmax(floor(at - h), 0.0)));
            x1 = min(x1, int(fmin(floor(at + h), double(g.g[0] - 1))));
          }
          if (rest >= 0.0 && x0 <= x1) {
            const int64_t row = (int64_t(z) * g.g[1] + y) * g.g[0];
            a = cell_start[row + x0];
            b = cell_start[row + x1 + 1];
          }
        }
        unsigned longs = __ballot_sync(0xffffffffu, b - a > FAR_RUN);
        bool own = true;                           // the lanes' own rows first
        do {
          int64_t i = a, last = b - a > FAR_RUN ? a : b;
          int step = 1;
          if (!own) {
            const int src = __ffs(longs) - 1;
            longs &= longs - 1;
            i = __shfl_sync(0xffffffffu, a, src) + lane;
            last = __shfl_sync(0xffffffffu, b, src);
            step = 32;
          }
          own = false;
          if (i < last) f(i, step, last);
          __syncwarp();
        } while (longs);
      }
    };
    int R = LANE_R;
    for (;; R *= 2) {
      long long have = 0;
      rows(min(R, rmax), INFINITY,
           [&](int64_t i, int step, int64_t last) { have += (last - i + step - 1) / step; });
      for (int off = 16; off > 0; off >>= 1) have += __shfl_xor_sync(0xffffffffu, have, off);
      if (have >= k || R >= rmax) break;
    }
    float s[K];
    int id[K];
    double r = INFINITY;
    for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
      for (int j = 0; j < K; ++j) { s[j] = INFINITY; id[j] = INT_MAX; }
      const float rf = __double2float_ru(r);
      rows(min(R, rmax), r, [&](int64_t i, int step, int64_t last) {
        // any k points bound the distance: of a long row the first pass takes its first few
        if (pass == 0 && step == 32) last = min(last, i - lane + FAR_FIRST * K);
        evals += max(int64_t(0), (last - i + step - 1) / step);
        float4 p4[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) p4[u] = pts[min(i + u * step, last - 1)];
        for (int u = 0; i < last; i += step) {
          const float4 p = u == 0 ? p4[0] : (u == 1 ? p4[1] : (u == 2 ? p4[2] : p4[3]));
          if (++u == 4) {                          // the next four, whose loads overlap
            u = 0;
#pragma unroll
            for (int v = 0; v < 4; ++v) p4[v] = pts[min(i + (v + 1) * step, last - 1)];
          }
          const int pid = __float_as_int(p.w);
          const float sd = __fsqrt_rn(sq_dist<D>(p, q));
          if (pid == qi || sd > rf || !key_less(sd, pid, s[K - 1], id[K - 1])) continue;
#pragma unroll
          for (int j = K - 1; j > 0; --j) {
            const bool lp = key_less(sd, pid, s[j - 1], id[j - 1]);
            const bool lc = key_less(sd, pid, s[j], id[j]);
            const float ns = lp ? s[j - 1] : (lc ? sd : s[j]);
            const int ni = lp ? id[j - 1] : (lc ? pid : id[j]);
            s[j] = ns;
            id[j] = ni;
          }
          if (key_less(sd, pid, s[0], id[0])) { s[0] = sd; id[0] = pid; }
        }
      });
      // the m smallest heads of the lanes' sorted lists, in order
      float last = INFINITY;
      for (int t = 0; t < m; ++t) {
        float bs = s[0];
        int bi = id[0];
        for (int off = 16; off > 0; off >>= 1) {
          const float os = __shfl_xor_sync(0xffffffffu, bs, off);
          const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
          if (key_less(os, oi, bs, bi)) { bs = os; bi = oi; }
        }
        if (id[0] == bi && s[0] == bs && bi != INT_MAX) {
#pragma unroll
          for (int j = 0; j + 1 < K; ++j) { s[j] = s[j + 1]; id[j] = id[j + 1]; }
          s[K - 1] = INFINITY;
          id[K - 1] = INT_MAX;
        }
        last = bs;
        if (pass == 1 && lane == 0) {
          out_idx[int64_t(qi) * k + 1 + t] = bi;
          out_dist[int64_t(qi) * k + 1 + t] = bs;
        }
      }
      // every point within r of the query lies in the cells within r (margin: float32 and FP64
      // rounding, as in the lane pass)
      r = double(last) * (1.0 + 8e-6) + 2.0 * g.eps_abs;
      const double need = r / g.cs + 1.0;
      R = isinf(last) || need >= double(rmax) ? rmax : max(1, int(need));
    }
    if (lane == 0) {
      out_idx[int64_t(qi) * k] = qi;
      out_dist[int64_t(qi) * k] = 0.f;
    }
  }
  for (int off = 16; off > 0; off >>= 1) evals += __shfl_xor_sync(0xffffffffu, evals, off);
  if (lane == 0 && evals) atomicAdd(&counters[0], evals);
}

// Radius search.  pass 0 counts into count[qi]; pass 1 writes (column, distance) from
// indptr[qi] in the same walk order.
template <int D>
__global__ void __launch_bounds__(SP_T)
sp_radius_kernel(const float4* __restrict__ pts, const int64_t* __restrict__ cell_start,
                 const SpGrid* __restrict__ G, int64_t n, float r2lo, float r2hi, int pass,
                 int32_t* __restrict__ count, const int64_t* __restrict__ indptr,
                 int32_t* __restrict__ col, float* __restrict__ val,
                 unsigned long long* __restrict__ counters) {
  const SpGrid g = *G;
  if (g.status) return;
  const int lane = threadIdx.x & 31;
  const int R = g.ring;
  unsigned long long evals = 0;
  for (int64_t pos = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; pos < n;
       pos += int64_t(gridDim.x) * blockDim.x) {
    const float4 q = pts[pos];
    const int qi = __float_as_int(q.w);
    const int cx = cell_axis(q.x, g, 0), cy = cell_axis(q.y, g, 1);
    const int cz = D == 3 ? cell_axis(q.z, g, 2) : 0;
    int64_t w = pass == 1 ? indptr[qi] : 0;
    int32_t cnt = 0;
    auto visit = [&](const float4& p) {
      const float d2 = sq_dist<D>(p, q);
      const int pid = __float_as_int(p.w);
      if (pid != qi && d2 <= r2hi && d2 >= r2lo) {
        if (pass == 1) {
          col[w] = pid;
          val[w] = __fsqrt_rn(d2);
          ++w;
        }
        ++cnt;
      }
    };
    const int zlo = D == 3 ? max(cz - R, 0) : 0, zhi = D == 3 ? min(cz + R, g.g[2] - 1) : 0;
    const int x0 = max(cx - R, 0), x1 = min(cx + R, g.g[0] - 1);
    for (int z = zlo; z <= zhi; ++z) {
      for (int y = max(cy - R, 0); y <= min(cy + R, g.g[1] - 1); ++y) {
        const int64_t row = (int64_t(z) * g.g[1] + y) * g.g[0];
        const int64_t a = cell_start[row + x0], b = cell_start[row + x1 + 1];
        evals += b - a;
        scan_run(pts, a, b, visit);
      }
    }
    if (pass == 0) count[qi] = cnt;
  }
  __syncwarp();
  for (int off = 16; off > 0; off >>= 1) evals += __shfl_xor_sync(0xffffffffu, evals, off);
  if (lane == 0) atomicAdd(&counters[0], evals);
}

// Columns of every row in ascending order (they are distinct within a row): the rank of an
// entry is the number of smaller columns in its row.  One warp per row.
__global__ void __launch_bounds__(SP_T)
sp_sort_rows_kernel(const int64_t* __restrict__ indptr, int64_t n, const int32_t* __restrict__ col_in,
                    const float* __restrict__ val_in, int32_t* __restrict__ col_out,
                    float* __restrict__ val_out) {
  __shared__ int32_t tile_all[SP_W][SORT_TILE];
  const int lane = threadIdx.x & 31;
  int32_t* tile = tile_all[threadIdx.x >> 5];
  const int64_t wid = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t row = wid; row < n; row += nw) {
    const int64_t a = indptr[row];
    const int64_t m = indptr[row + 1] - a;
    if (m <= 32) {                                      // one entry a lane
      const int32_t mine = lane < m ? col_in[a + lane] : INT_MAX;
      const float v = lane < m ? val_in[a + lane] : 0.f;
      int rank = 0;
      for (int t = 0; t < int(m); ++t) rank += __shfl_sync(0xffffffffu, mine, t) < mine;
      if (lane < m) {
        col_out[a + rank] = mine;
        val_out[a + rank] = v;
      }
      continue;
    }
    for (int64_t g0 = 0; g0 < m; g0 += 32 * SORT_E) {
      int32_t mine[SORT_E];
      int64_t rank[SORT_E];
#pragma unroll
      for (int e = 0; e < SORT_E; ++e) {
        const int64_t j = g0 + lane + 32 * e;
        mine[e] = j < m ? col_in[a + j] : INT_MAX;
        rank[e] = 0;
      }
      for (int64_t t0 = 0; t0 < m; t0 += SORT_TILE) {
        const int cnt = int(imin64(SORT_TILE, m - t0));
        __syncwarp();
        for (int j = lane; j < cnt; j += 32) tile[j] = col_in[a + t0 + j];
        __syncwarp();
        for (int t = 0; t < cnt; ++t) {
          const int32_t v = tile[t];
#pragma unroll
          for (int e = 0; e < SORT_E; ++e) rank[e] += v < mine[e];
        }
      }
#pragma unroll
      for (int e = 0; e < SORT_E; ++e) {
        const int64_t j = g0 + lane + 32 * e;
        if (j < m) {
          col_out[a + rank[e]] = mine[e];
          val_out[a + rank[e]] = val_in[a + j];
        }
      }
    }
  }
}

// FP64 edge lengths of a CSR graph from float64 coordinates (gr.py:32-34): squares summed axis
// by axis in order, correctly rounded sqrt.  One warp per row.
__global__ void sp_edge_len_kernel(const double* __restrict__ X, int d,
                                   const int64_t* __restrict__ indptr, int64_t n,
                                   const int32_t* __restrict__ cols, double* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t wid = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t row = wid; row < n; row += nw) {
    const double* xi = X + row * d;
    for (int64_t e = indptr[row] + lane; e < indptr[row + 1]; e += 32) {
      const double* xj = X + int64_t(cols[e]) * d;
      double acc = 0;
      for (int a = 0; a < d; ++a) {
        const double t = __dsub_rn(xi[a], xj[a]);
        const double t2 = __dmul_rn(t, t);
        acc = a == 0 ? t2 : __dadd_rn(acc, t2);
      }
      out[e] = __dsqrt_rn(acc);
    }
  }
}

__global__ void sp_init_kernel(unsigned* mm, unsigned long long* nonfinite,
                               unsigned long long* counters, int32_t* n_far) {
  if (threadIdx.x < 3) { mm[threadIdx.x] = 0xffffffffu; mm[3 + threadIdx.x] = 0u; }
  if (threadIdx.x == 0) { *nonfinite = 0; *n_far = 0; counters[0] = 0; counters[1] = 0; }
}

__global__ void sp_stats_kernel(const SpGrid* __restrict__ G, const unsigned long long* __restrict__ nonfinite,
                                const unsigned long long* __restrict__ counters, int64_t n,
                                int64_t* __restrict__ stats) {
  if (threadIdx.x != 0) return;
  const SpGrid g = *G;
  stats[MSC_SP_STAT_NONFINITE] = int64_t(*nonfinite);
  stats[MSC_SP_STAT_STATUS] = g.status;
  stats[MSC_SP_STAT_CELLS] = g.status ? 0 : g.ncells;
  stats[MSC_SP_STAT_CHUNKS] = g.status ? 0 : (n + 31) / 32;
  stats[MSC_SP_STAT_EVALS] = int64_t(counters[0]);
  stats[MSC_SP_STAT_EXPANDED] = int64_t(counters[1]);
  stats[MSC_SP_STAT_RING] = g.status ? 0 : g.ring;
  stats[MSC_SP_STAT_CELL_SIDE] = g.status ? 0 : int64_t(__double_as_longlong(g.cs));
}

struct SpWs {
  SpGrid* G;
  unsigned* mm;
  unsigned long long* nonfinite;
  unsigned long long* counters;
  int64_t* cell;          // [n]
  int32_t* count;         // [cap]
  int32_t* cursor;        // [cap], right behind count
  int64_t* cell_start;    // [cap + 1]
  int64_t* scan_scratch;
  float4* pts;            // [n]
  int32_t* far_rows;      // [n] queries of the warp pass
  int32_t* n_far;
};

int64_t cell_cap(int64_t n) { return 4 * n + 16; }

SpWs carve(Carver& c, int64_t n) {
  const int64_t cap = cell_cap(n);
  SpWs w;
  w.G = c.take<SpGrid>(1);
  w.mm = c.take<unsigned>(8);
  w.nonfinite = c.take<unsigned long long>(1);
  w.counters = c.take<unsigned long long>(2);
  w.cell = c.take<int64_t>(n);
  w.count = c.take<int32_t>(cap);
  w.cursor = c.take<int32_t>(cap);
  w.cell_start = c.take<int64_t>(cap + 1);
  w.scan_scratch = c.take<int64_t>(scan_i32_scratch_elems(cap));
  w.pts = c.take<float4>(n);
  w.far_rows = c.take<int32_t>(n);
  w.n_far = c.take<int32_t>(1);
  return w;
}


unsigned flat_grid(int64_t items, int threads) {
  const int64_t b = (items + threads - 1) / threads;
  return unsigned(std::max<int64_t>(1, std::min<int64_t>(b, int64_t(num_sms()) * 16)));
}

// The grid: bounding box, plan, binning, cell-ordered points.  The cell table is sized
// for the cap; the plan never uses more cells than that.
int build_grid(const float* X, int64_t n, int d, int mode, int k, double reach, const SpWs& w,
               cudaStream_t st) {
  const int64_t cap = cell_cap(n);
  sp_init_kernel<<<1, 32, 0, st>>>(w.mm, w.nonfinite, w.counters, w.n_far);
  MSC_LAUNCH_CHECK();
  sp_bbox_kernel<<<flat_grid(n, 256), 256, 0, st>>>(X, n, d, w.mm, w.nonfinite);
  MSC_LAUNCH_CHECK();
  sp_plan_kernel<<<1, 32, 0, st>>>(w.mm, w.nonfinite, n, d, mode, k, reach, w.G);
  MSC_LAUNCH_CHECK();
  // counts and cursors lie one behind the other: one memset
  MSC_CUDA_TRY(cudaMemsetAsync(w.count, 0, reinterpret_cast<char*>(w.cursor + cap) -
                                               reinterpret_cast<char*>(w.count), st));
  sp_bin_kernel<<<flat_grid(n, 256), 256, 0, st>>>(X, n, d, w.G, w.cell, w.count);
  MSC_LAUNCH_CHECK();
  // a scan over the whole cap: cells the plan does not use hold zero counts, so
  // cell_start[ncells] = n
  MSC_TRY(scan_excl_i32(w.count, cap, w.cell_start, w.scan_scratch, st));
  sp_place_kernel<<<flat_grid(n, 256), 256, 0, st>>>(X, n, d, w.G, w.cell, w.cell_start, w.cursor,
                                                      w.pts);
  MSC_LAUNCH_CHECK();
  return MSC_OK;
}

// one lane per query; as many blocks as there are queries, up to four waves of full SMs
unsigned search_grid(int64_t n) {
  const int64_t blocks = (n + SP_T - 1) / SP_T;
  return unsigned(std::max<int64_t>(1, std::min<int64_t>(blocks, int64_t(num_sms()) * 64)));
}

template <int K>
int launch_knn_k(const SpWs& w, int64_t n, int d, int k, int32_t* idx, float* dist, cudaStream_t st) {
  if (d == 2)
    sp_knn_kernel<K, 2><<<search_grid(n), SP_T, 0, st>>>(w.pts, w.cell_start, w.G, n, k, idx,
                                                         dist, w.counters, w.far_rows, w.n_far);
  else
    sp_knn_kernel<K, 3><<<search_grid(n), SP_T, 0, st>>>(w.pts, w.cell_start, w.G, n, k, idx,
                                                         dist, w.counters, w.far_rows, w.n_far);
  MSC_LAUNCH_CHECK();
  const unsigned gf = search_grid(std::min<int64_t>(n * 32, int64_t(num_sms()) * 16 * SP_T));
  if (d == 2)
    sp_knn_far_kernel<K, 2><<<gf, SP_T, 0, st>>>(w.pts, w.cell_start, w.G, k, w.far_rows, w.n_far,
                                                 idx, dist, w.counters);
  else
    sp_knn_far_kernel<K, 3><<<gf, SP_T, 0, st>>>(w.pts, w.cell_start, w.G, k, w.far_rows, w.n_far,
                                                 idx, dist, w.counters);
  MSC_LAUNCH_CHECK();
  return MSC_OK;
}

}  // namespace

size_t spatial_knn_workspace_bytes(int64_t n) {
  Carver c(nullptr);
  carve(c, n);
  return c.bytes();
}

int launch_spatial_knn(const float* X, int64_t n, int d, int k, int32_t* idx, float* dist,
                       int64_t* stats, void* ws, cudaStream_t st) {
  Carver c(ws);
  const SpWs w = carve(c, n);
  MSC_TRY(build_grid(X, n, d, 0, k, 0.0, w, st));
  const int m = k - 1;
  if (m <= 8) MSC_TRY(launch_knn_k<8>(w, n, d, k, idx, dist, st));
  else if (m <= 16) MSC_TRY(launch_knn_k<16>(w, n, d, k, idx, dist, st));
  else if (m <= 32) MSC_TRY(launch_knn_k<32>(w, n, d, k, idx, dist, st));
  else MSC_TRY(launch_knn_k<64>(w, n, d, k, idx, dist, st));
  sp_stats_kernel<<<1, 32, 0, st>>>(w.G, w.nonfinite, w.counters, n, stats);
  MSC_LAUNCH_CHECK();
  return MSC_OK;
}

size_t spatial_radius_workspace_bytes(int64_t n) {
  Carver c(nullptr);
  carve(c, n);
  c.take<int32_t>(n);                     // per-row counts
  return c.bytes();
}

int launch_spatial_radius_count(const float* X, int64_t n, int d, double radius, double min_radius,
                                int64_t* indptr, int64_t* stats, void* ws, cudaStream_t st) {
  Carver c(ws);
  const SpWs w = carve(c, n);
  int32_t* rowcnt = c.take<int32_t>(n);
  const double reach = radius * (1.0 + 1e-6);
  MSC_TRY(build_grid(X, n, d, 1, 0, reach, w, st));
  MSC_CUDA_TRY(cudaMemsetAsync(rowcnt, 0, sizeof(int32_t) * n, st));
  const float r2hi = float(radius * radius), r2lo = float(min_radius * min_radius);
  if (d == 2)
    sp_radius_kernel<2><<<search_grid(n), SP_T, 0, st>>>(w.pts, w.cell_start, w.G, n, r2lo,
                                                         r2hi, 0, rowcnt, nullptr, nullptr,
                                                         nullptr, w.counters);
  else
    sp_radius_kernel<3><<<search_grid(n), SP_T, 0, st>>>(w.pts, w.cell_start, w.G, n, r2lo,
                                                         r2hi, 0, rowcnt, nullptr, nullptr,
                                                         nullptr, w.counters);
  MSC_LAUNCH_CHECK();
  MSC_TRY(scan_excl_i32(rowcnt, n, indptr, w.scan_scratch, st));
  sp_stats_kernel<<<1, 32, 0, st>>>(w.G, w.nonfinite, w.counters, n, stats);
  MSC_LAUNCH_CHECK();
  return MSC_OK;
}

size_t spatial_radius_fill_scratch_bytes(int64_t nnz) {
  Carver c(nullptr);
  c.take<int32_t>(nnz);
  c.take<float>(nnz);
  return c.bytes();
}

int launch_spatial_radius_fill(int64_t n, int d, double radius, double min_radius,
                               const int64_t* indptr, int64_t nnz, int32_t* cols, float* dist,
                               void* ws, void* scratch, cudaStream_t st) {
  Carver c(ws);
  const SpWs w = carve(c, n);
  Carver s(scratch);
  int32_t* col_tmp = s.take<int32_t>(nnz);
  float* val_tmp = s.take<float>(nnz);
  const float r2hi = float(radius * radius), r2lo = float(min_radius * min_radius);
  if (nnz > 0) {
    if (d == 2)
      sp_radius_kernel<2><<<search_grid(n), SP_T, 0, st>>>(w.pts, w.cell_start, w.G, n, r2lo,
                                                           r2hi, 1, nullptr, indptr, col_tmp,
                                                           val_tmp, w.counters);
    else
      sp_radius_kernel<3><<<search_grid(n), SP_T, 0, st>>>(w.pts, w.cell_start, w.G, n, r2lo,
                                                           r2hi, 1, nullptr, indptr, col_tmp,
                                                           val_tmp, w.counters);
    MSC_LAUNCH_CHECK();
    sp_sort_rows_kernel<<<search_grid(n * 32), SP_T, 0, st>>>(indptr, n, col_tmp, val_tmp, cols,
                                                             dist);
    MSC_LAUNCH_CHECK();
  }
  return MSC_OK;
}

int launch_spatial_edge_lengths(const double* X, int64_t n, int d, const int64_t* indptr,
                                const int32_t* cols, double* out, cudaStream_t st) {
  sp_edge_len_kernel<<<flat_grid(n * 32, 256), 256, 0, st>>>(X, d, indptr, n, cols, out);
  MSC_LAUNCH_CHECK();
  return MSC_OK;
}

}  // namespace msc
