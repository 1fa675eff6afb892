// Edge preparation of the UMAP layout, on the device, from a connectivities CSR that is already in
// HBM (the hand-off from the neighbour graph to its first consumer, without a host round trip).
//
// Reference: metalsinglecell embedding.py.  `umap()` first drops the edges too weak to be sampled
// once over the run (`_prune_weak_edges`, embedding.py:255-267: keep w >= max(w) / n_epochs, the
// division in float32 — NumPy 2 keeps a float32 scalar divided by a Python float in float32), then
// takes the kept graph as COO in CSR order (`graph.tocoo()`, embedding.py:115) and derives each
// edge's sampling period (`_make_epochs_per_sample`, embedding.py:123-137, in FP64:
// n_epochs / (n_epochs · (w / max w)), -1 for an edge never sampled).
//
// Kernels: (1) the largest weight (a max of non-negative float32 values, exact in any order);
// (2) kept entries per block of rows, and by the last block to finish their prefix sums; (3) per
// block of rows, the kept entries compacted in their CSR order with their row, column, weight and
// period, and the kept graph's row pointers.
//
// The entries' bytes bound it (8 read, 20 written each); what it spent its time on instead were the
// chains of loads of a warp that takes one row of some twenty entries at a time.  Here a block
// takes EB_ROWS rows' entries as one flat range, so all lanes load and every load is coalesced; an
// entry finds its row by a search of the block's row pointers in shared memory.  200,000 rows of
// 22 entries, a warp per row / this: counting and scanning 33 / 17 us, compacting 63 / 41.  The
// compaction is now bound by its instructions, above all the two FP64 divisions and the search.
#include "kernels.cuh"

namespace msc {

namespace {

constexpr int EB_THREADS = 256;
constexpr int EB_WARPS = EB_THREADS / 32;
constexpr int EB_ROWS = 64;       // rows a block: about 1400 entries at 15 neighbours
constexpr int EB_UNROLL = 4;      // entries a thread has in flight
constexpr int EB_CHUNK = EB_THREADS * EB_UNROLL;
static_assert(EB_CHUNK == 32 * 32, "a chunk's ballots fill one warp's lanes");

__global__ void weight_max_kernel(const float* __restrict__ data, const int64_t* __restrict__ nnz,
                                  unsigned* __restrict__ wmax_bits) {
  const int64_t m = *nnz;
  float mx = 0.f;
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < m;
       e += int64_t(gridDim.x) * blockDim.x)
    mx = fmaxf(mx, data[e]);
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(FULL, mx, o));
  if (lane_id() == 0 && mx > 0.f) atomic_max_nonneg(wmax_bits, mx);
}

__device__ __forceinline__ float keep_threshold(const unsigned* wmax_bits, int n_epochs) {
  return __fdiv_rn(__uint_as_float(*wmax_bits), float(n_epochs));
}

// Kept entries of each block of rows; the block that finishes last replaces the counts by their
// exclusive prefix sums (part[blocks]: the total).
__global__ void __launch_bounds__(EB_THREADS)
kept_count_kernel(const int64_t* __restrict__ indptr, const float* __restrict__ data, int64_t n,
                  int64_t blocks, int n_epochs, const unsigned* __restrict__ wmax_bits,
                  int64_t* __restrict__ part, unsigned* __restrict__ done) {
  __shared__ int64_t sums[EB_WARPS];
  __shared__ bool last;
  const float thr = keep_threshold(wmax_bits, n_epochs);
  const int lane = lane_id(), w = warp_id();
  for (int64_t b = blockIdx.x; b < blocks; b += gridDim.x) {
    const int64_t e0 = indptr[b * EB_ROWS], e1 = indptr[min64(n, (b + 1) * EB_ROWS)];
    int64_t c = 0;
    for (int64_t c0 = e0; c0 < e1; c0 += EB_CHUNK) {
      const float* w0 = data + c0 + threadIdx.x;
      const int left = int(min64(e1 - c0, EB_CHUNK)) - int(threadIdx.x);
      float v[EB_UNROLL];
#pragma unroll
      for (int u = 0; u < EB_UNROLL; ++u) v[u] = u * EB_THREADS < left ? w0[u * EB_THREADS] : 0.f;
      int m = 0;
#pragma unroll
      for (int u = 0; u < EB_UNROLL; ++u) m += u * EB_THREADS < left && v[u] >= thr ? 1 : 0;
      c += m;
    }
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(FULL, c, o);
    if (lane == 0) sums[w] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int j = 1; j < EB_WARPS; ++j) c += sums[j];
      part[b] = c;
    }
    __syncthreads();
  }
  __threadfence();
  if (threadIdx.x == 0) last = atomicAdd(done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  int64_t base = 0;
  for (int64_t b0 = 0; b0 < blocks; b0 += EB_CHUNK) {
    // four neighbouring counts a thread
    const int64_t b = b0 + int64_t(threadIdx.x) * EB_UNROLL;
    int64_t v[EB_UNROLL], t = 0;
#pragma unroll
    for (int u = 0; u < EB_UNROLL; ++u) {
      v[u] = t;
      t += b + u < blocks ? __ldcg(part + b + u) : 0;
    }
    int64_t x = t;
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(FULL, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) sums[w] = x;
    __syncthreads();
    int64_t before = base, all = 0;
    for (int j = 0; j < EB_WARPS; ++j) {
      if (j < w) before += sums[j];
      all += sums[j];
    }
#pragma unroll
    for (int u = 0; u < EB_UNROLL; ++u)
      if (b + u < blocks) part[b + u] = before + x - t + v[u];
    base += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blocks] = base;
}

__global__ void __launch_bounds__(EB_THREADS)
compact_kernel(const int64_t* __restrict__ indptr, const int32_t* __restrict__ indices,
               const float* __restrict__ data, int64_t n, int64_t blocks, int n_epochs,
               const unsigned* __restrict__ wmax_bits, const int64_t* __restrict__ part,
               int64_t* __restrict__ out_ptr, int32_t* __restrict__ rows,
               int32_t* __restrict__ cols, float* __restrict__ weights,
               double* __restrict__ eps) {
  __shared__ int64_t ptr[EB_ROWS + 1];
  __shared__ int at[EB_ROWS];             // where in the chunk the rows start (-1: before it)
  __shared__ unsigned ballots[32];        // word u * EB_WARPS + w: 32 neighbouring entries
  const float thr = keep_threshold(wmax_bits, n_epochs);
  // the kept graph's largest weight is the input's (the largest entry is always kept)
  const double wmax = double(__uint_as_float(*wmax_bits));
  const double ne = double(n_epochs);
  const int lane = lane_id(), w = warp_id();
  for (int64_t b = blockIdx.x; b < blocks; b += gridDim.x) {
    const int64_t r0 = b * EB_ROWS;
    const int nr = int(min64(n - r0, EB_ROWS));
    __syncthreads();                       // ptr of the block before
    if (threadIdx.x <= nr) ptr[threadIdx.x] = indptr[r0 + threadIdx.x];
    int64_t o = part[b];
    __syncthreads();
    const int64_t e0 = ptr[0], e1 = ptr[nr];
    for (int64_t c0 = e0; c0 < e1; c0 += EB_CHUNK) {
      const float* w0 = data + c0 + threadIdx.x;
      const int32_t* i0 = indices + c0 + threadIdx.x;
      const int len = int(min64(e1 - c0, EB_CHUNK)), left = len - int(threadIdx.x);
      float v[EB_UNROLL];
      int32_t col[EB_UNROLL];
      unsigned m[EB_UNROLL];
#pragma unroll
      for (int u = 0; u < EB_UNROLL; ++u) {
        const bool in = u * EB_THREADS < left;
        v[u] = in ? w0[u * EB_THREADS] : 0.f;
        col[u] = in ? i0[u * EB_THREADS] : 0;
      }
      if (threadIdx.x < nr)
        at[threadIdx.x] = ptr[threadIdx.x] < c0 ? -1 : int(min64(ptr[threadIdx.x] - c0, EB_CHUNK));
#pragma unroll
      for (int u = 0; u < EB_UNROLL; ++u) {
        m[u] = __ballot_sync(FULL, u * EB_THREADS < left && v[u] >= thr);
        if (lane == 0) ballots[u * EB_WARPS + w] = m[u];
      }
      __syncthreads();
      const unsigned mine = ballots[lane];
      int exc = __popc(mine);
      for (int s = 1; s < 32; s <<= 1) {
        const int y = __shfl_up_sync(FULL, exc, s);
        if (lane >= s) exc += y;
      }
      const int total = __shfl_sync(FULL, exc, 31);
      exc -= __popc(mine);
      int32_t* rows_o = rows + o;
      int32_t* cols_o = cols + o;
      float* w_o = weights + o;
      double* eps_o = eps + o;
#pragma unroll
      for (int u = 0; u < EB_UNROLL; ++u) {
        const int before = __shfl_sync(FULL, exc, u * EB_WARPS + w);
        if (m[u] >> lane & 1) {
          const int e = u * EB_THREADS + int(threadIdx.x);
          int lo = 0;                      // the last row that starts at or before e
#pragma unroll
          for (int s = EB_ROWS / 2; s > 0; s >>= 1)
            if (lo + s < nr && at[lo + s] <= e) lo += s;
          const int p = before + __popc(m[u] & ((1u << lane) - 1u));
          rows_o[p] = int32_t(r0) + lo;
          cols_o[p] = col[u];
          w_o[p] = v[u];
          const double ns = __dmul_rn(ne, __ddiv_rn(double(v[u]), wmax));
          eps_o[p] = ns > 0.0 ? __ddiv_rn(ne, ns) : -1.0;
        }
      }
      // row pointers of the rows that start in this chunk (a lane each)
      if (w < EB_ROWS / 32) {
        const int r = w * 32 + lane;
        const int x = r < nr ? at[r] : -1;
        const bool here = x >= 0 && x < len;
        const unsigned bits = __shfl_sync(FULL, mine, here ? x >> 5 : 0);
        const int ex = __shfl_sync(FULL, exc, here ? x >> 5 : 0);
        if (here) out_ptr[r0 + r] = o + ex + __popc(bits & ((1u << (x & 31)) - 1u));
      }
      o += total;
      __syncthreads();                     // at and ballots, before the next chunk
    }
    // the rows that start at the block's end (empty ones), and behind the last block the total
    for (int r = threadIdx.x; r < nr; r += EB_THREADS)
      if (ptr[r] >= e1) out_ptr[r0 + r] = o;
    if (b == blocks - 1 && threadIdx.x == 0) out_ptr[n] = o;
  }
}

struct EdgeWs {
  unsigned* wmax;                // [0] the largest weight's bits, [1] blocks that have counted
  int64_t* part;
};

int64_t edge_blocks(int64_t n) { return ceil_div(n, EB_ROWS); }

EdgeWs carve_edges(Carver& c, int64_t n) {
  EdgeWs w;
  w.wmax = c.take<unsigned>(8);
  w.part = c.take<int64_t>(edge_blocks(n) + 1);
  return w;
}

}  // namespace

size_t umap_edges_workspace_bytes(int64_t n) {
  Carver c(nullptr);
  carve_edges(c, n);
  return c.bytes();
}

int launch_umap_edges(const int64_t* indptr, const int32_t* indices, const float* data, int64_t n,
                      int n_epochs, int64_t* out_ptr, int32_t* rows, int32_t* cols,
                      float* weights, double* eps, void* ws, cudaStream_t st) {
  Carver c(ws);
  EdgeWs w = carve_edges(c, n);
  MSC_CUDA_TRY(cudaMemsetAsync(w.wmax, 0, 2 * sizeof(unsigned), st));
  const int sms = num_sms();
  weight_max_kernel<<<sms * 4, 256, 0, st>>>(data, indptr + n, w.wmax);
  MSC_LAUNCH_CHECK();
  const int64_t blocks = edge_blocks(n);
  const int g = int(std::min<int64_t>(blocks, int64_t(sms) * 64));
  kept_count_kernel<<<g, EB_THREADS, 0, st>>>(indptr, data, n, blocks, n_epochs, w.wmax, w.part,
                                              w.wmax + 1);
  MSC_LAUNCH_CHECK();
  compact_kernel<<<g, EB_THREADS, 0, st>>>(indptr, indices, data, n, blocks, n_epochs, w.wmax,
                                           w.part, out_ptr, rows, cols, weights, eps);
  MSC_LAUNCH_CHECK();
  return MSC_OK;
}

}  // namespace msc
