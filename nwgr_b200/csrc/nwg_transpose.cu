// Whether a graph's in-CSR is the transpose of its out-CSR, for the callers
// whose results are defined on the out-graph alone but that run faster over
// both: betweenness and the device verifier.  Registration leaves the
// transpose to its caller (host arrays are checked on request, device arrays
// never), and a graph registered without an in-CSR may in fact be directed.
//
// The two CSRs are compared as multisets of edges by a 64-bit hash sum, so
// rows may be in any order; once per graph.  Every warp has an equal part of the
// edges and finds its first row by one search, so hubs need no list of pieces
// and the comparison no memory but the sum, which is in the registration
// tables (with a list and a sum allocated and freed, a verification's first
// call took up to 20 ms longer where the host was busy).
#include <algorithm>

#include "nwg_internal.cuh"

namespace nwg {
namespace {

constexpr int      kTrThreads = 256;
constexpr uint64_t kTrMin     = 64;  // edges a warp takes at least

__device__ __forceinline__ unsigned long long tr_block_sum(unsigned long long x) {
  __shared__ unsigned long long red[kTrThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(kFullMask, x, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
  __syncthreads();
  unsigned long long t = 0;
#pragma unroll
  for (int i = 0; i < kTrThreads / 32; ++i) t += red[i];
  return t;
}

// splitmix64's finalizer (Steele, Lea and Flood 2014).
__device__ __forceinline__ uint64_t tr_mix(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// Adds a hash of every edge (mode 0: row -> column), takes away that of every
// reversed edge (1), or both (2): over a CSR and its transpose the sum is
// zero, whatever the order of their rows.  A warp takes edges [lo, hi): 32 rows
// at a time, whose edges its lanes read in order, each finding its edge's row
// by five steps over the lanes' row starts; behind 32 empty rows it searches
// again.  With a lane per short row RMAT-22 (130M entries) took 0.87 ms,
// 0.57 so.
__global__ void __launch_bounds__(kTrThreads) k_tr_edge_hash(const uint64_t* __restrict__ off,
                                                             const uint32_t* __restrict__ col, uint64_t n, uint64_t m,
                                                             uint64_t per_warp, uint32_t mode,
                                                             unsigned long long* sum) {
  constexpr int      kEdges = 4;  // a lane's loads in flight
  const unsigned     lane   = threadIdx.x & 31;
  const uint64_t     warp   = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t     lo = min(m, warp * per_warp), hi = min(m, lo + per_warp);
  const uint32_t     span = (uint32_t)(hi - lo);
  unsigned long long h    = 0;
  auto row_of = [&](uint64_t i) {  // the row that holds edge i
    uint64_t row = 0, end = n;     // off[row] <= i < off[end]
    while (end - row > 1) {
      const uint64_t mid = (row + end) >> 1;
      if (off[mid] <= i) row = mid;
      else end = mid;
    }
    return row;
  };
  if (lo < hi) {
    for (uint64_t row = row_of(lo); row < n;) {
      const uint32_t at = row + lane < n ? (uint32_t)(min(hi, max(lo, off[row + lane])) - lo) : span;
      const uint32_t from = __shfl_sync(kFullMask, at, 0);
      const uint32_t to   = (uint32_t)(min(hi, max(lo, off[min(n, row + 32)])) - lo);
      for (uint32_t i0 = from; i0 < to; i0 += 32 * kEdges) {
        uint32_t v[kEdges];
#pragma unroll
        for (int k = 0; k < kEdges; ++k) {
          const uint32_t i = i0 + k * 32 + lane;
          v[k]             = i < to ? __ldg(col + lo + i) : 0u;
        }
#pragma unroll
        for (int k = 0; k < kEdges; ++k) {
          const uint32_t i = i0 + k * 32 + lane;
          uint32_t       o = 0;  // the last row that starts at i or before
#pragma unroll
          for (int s = 16; s >= 1; s >>= 1)
            if (__shfl_sync(kFullMask, at, o + s) <= i) o += s;
          if (i >= to) continue;
          const uint64_t u = row + o;
          if (mode != 1) h += tr_mix((u << 32) | v[k]);
          if (mode != 0) h -= tr_mix(((uint64_t)v[k] << 32) | u);
        }
      }
      if (to >= span) break;  // every later row starts at hi or after
      row += 32;
      if (from == to) row = max(row, row_of(lo + to));
    }
  }
  h = tr_block_sum(h);
  if (threadIdx.x == 0) atomicAdd(sum, h);
}

// The comparison itself, on `stream`, which it synchronises.
int compare_csrs(const GraphDev* g, cudaStream_t stream, bool* same) {
  *same = false;
  if (g->in_m != g->m) return NWG_OK;
  const bool          one   = g->in_off == g->off && g->in_col == g->col;
  const uint64_t      warps = (uint64_t)g->sm_count * 8 * (kTrThreads / 32);
  const uint64_t      per   = std::max(kTrMin, (g->m + warps - 1) / warps);
  const uint64_t      used  = (g->m + per - 1) / per;
  const int           grid  = (int)std::max<uint64_t>(1, (used * 32 + kTrThreads - 1) / kTrThreads);
  unsigned long long* sum   = reinterpret_cast<unsigned long long*>(g->tables);
  unsigned long long  h     = 1;
  NWG_CUDA_TRY(cudaMemsetAsync(sum, 0, sizeof h, stream));
  k_tr_edge_hash<<<grid, kTrThreads, 0, stream>>>(g->off, g->col, g->n, g->m, per, one ? 2u : 0u, sum);
  if (!one) k_tr_edge_hash<<<grid, kTrThreads, 0, stream>>>(g->in_off, g->in_col, g->n, g->m, per, 1u, sum);
  NWG_CUDA_TRY(cudaGetLastError());
  NWG_CUDA_TRY(cudaMemcpyAsync(&h, sum, sizeof h, cudaMemcpyDeviceToHost, stream));
  NWG_CUDA_TRY(cudaStreamSynchronize(stream));
  *same = h == 0;
  return NWG_OK;
}

}  // namespace

// Whether the in-CSR holds the out-CSR's edges, reversed; compared on a
// graph's first call, on the current device and `stream`.
int csrs_transposed(GraphDev* g, cudaStream_t stream, bool* yes) {
  std::lock_guard<std::mutex> lk(g->transposed_mu);
  if (g->transposed < 0) {
    bool      same = false;
    const int rc   = compare_csrs(g, stream, &same);
    if (rc) return rc;
    g->transposed = same ? 1 : 0;
  }
  *yes = g->transposed == 1;
  return NWG_OK;
}

}  // namespace nwg
