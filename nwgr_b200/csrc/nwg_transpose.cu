// Whether a graph's in-CSR is the transpose of its out-CSR, for the callers
// whose results are defined on the out-graph alone but that run faster over
// both: betweenness and the device verifier.  Registration leaves the
// transpose to its caller (host arrays are checked on request, device arrays
// never), and a graph registered without an in-CSR may in fact be directed.
//
// The two CSRs are compared as multisets of edges by a 64-bit hash sum, so
// rows may be in any order: 0.2 ms on RMAT-20 (32M entries), once per graph.
#include <algorithm>
#include <string>

#include "nwg_internal.cuh"

namespace nwg {
namespace {

constexpr int kTrThreads = 256;

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
// zero, whatever the order of their rows.  Eight lanes a vertex; vertices of
// more than kHubPiece edges by their pieces, a warp each.
__global__ void __launch_bounds__(kTrThreads) k_tr_edge_hash(const uint64_t* __restrict__ off,
                                                             const uint32_t* __restrict__ col, uint64_t n,
                                                             const uint64_t* __restrict__ piece, uint64_t npiece,
                                                             uint32_t mode, unsigned long long* sum) {
  const unsigned     lane  = threadIdx.x & 31;
  const uint64_t     warp  = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t     nwarp = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  unsigned long long h     = 0;
  auto edge = [&](uint64_t u, uint64_t v) {
    if (mode != 1) h += tr_mix((u << 32) | v);
    if (mode != 0) h -= tr_mix((v << 32) | u);
  };
  for (uint64_t i = warp * 4 + (lane >> 3); i < n; i += nwarp * 4) {
    const uint64_t e = off[i], end = off[i + 1];
    if (end - e > kHubPiece) continue;
    for (uint64_t j = e + (lane & 7); j < end; j += 8) edge(i, __ldg(col + j));
  }
  for (uint64_t i = warp; i < npiece; i += nwarp) {
    const uint64_t u  = piece[i] >> 32;
    const uint64_t b  = off[u] + (uint64_t)(uint32_t)piece[i] * kHubPiece;
    const uint64_t en = min(off[u + 1], b + kHubPiece);
    for (uint64_t j = b + lane; j < en; j += 32) edge(u, __ldg(col + j));
  }
  h = tr_block_sum(h);
  if (threadIdx.x == 0) atomicAdd(sum, h);
}

// The pieces of every vertex of more than kHubPiece edges.
__global__ void __launch_bounds__(kTrThreads) k_tr_pieces(const uint64_t* __restrict__ off, uint64_t n,
                                                          uint64_t* piece, uint64_t cap, unsigned long long* count) {
  const unsigned lane  = threadIdx.x & 31;
  const uint64_t nwarp = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < (n + 31) / 32; w += nwarp) {
    const uint64_t v    = w * 32 + lane;
    const uint64_t d    = v < n ? off[v + 1] - off[v] : 0;
    unsigned       hubs = __ballot_sync(kFullMask, d > kHubPiece);
    while (hubs) {
      const int src = __ffs(hubs) - 1;
      hubs &= hubs - 1;
      const uint64_t     np   = (__shfl_sync(kFullMask, d, src) + kHubPiece - 1) / kHubPiece;
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(count, (unsigned long long)np);
      base = __shfl_sync(kFullMask, base, 0);
      for (uint64_t j = lane; j < np; j += 32)
        if (base + j < cap) piece[base + j] = ((w * 32 + src) << 32) | j;
    }
  }
}

int grid_tr(const GraphDev* g, uint64_t items, uint64_t per_block) {
  const uint64_t want = (items + per_block - 1) / per_block;
  return (int)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)g->sm_count * 8, want));
}

// The comparison itself; synchronises.
int compare_csrs(const GraphDev* g, bool* same) {
  const bool one_off = g->in_off == g->off, one = one_off && g->in_col == g->col;
  *same              = false;
  if (g->in_m != g->m) return NWG_OK;
  struct Pieces {
    uint64_t* p = nullptr;
    uint64_t  n = 0;
    ~Pieces() { cudaFree(p); }
  } out, in;
  struct Stream {
    cudaStream_t        s   = nullptr;
    unsigned long long* sum = nullptr;
    ~Stream() {
      if (s) cudaStreamSynchronize(s);
      cudaFree(sum);
      if (s) cudaStreamDestroy(s);
    }
  } on;
  NWG_CUDA_TRY(cudaStreamCreateWithFlags(&on.s, cudaStreamNonBlocking));
  NWG_CUDA_TRY(cudaMalloc(&on.sum, sizeof *on.sum));
  int rc = hub_pieces(g, g->off, g->m, on.s, &out.p, &out.n);
  if (!rc && !one_off) rc = hub_pieces(g, g->in_off, g->in_m, on.s, &in.p, &in.n);
  if (rc) return rc;
  const int          grid = grid_tr(g, std::max(g->n, g->m / 8), kTrThreads / 8);
  unsigned long long h    = 1;
  NWG_CUDA_TRY(cudaMemsetAsync(on.sum, 0, sizeof h, on.s));
  k_tr_edge_hash<<<grid, kTrThreads, 0, on.s>>>(g->off, g->col, g->n, out.p, out.n, one ? 2u : 0u, on.sum);
  if (!one) {
    const Pieces& x = one_off ? out : in;
    k_tr_edge_hash<<<grid, kTrThreads, 0, on.s>>>(g->in_off, g->in_col, g->n, x.p, x.n, 1u, on.sum);
  }
  NWG_CUDA_TRY(cudaGetLastError());
  NWG_CUDA_TRY(cudaMemcpyAsync(&h, on.sum, sizeof h, cudaMemcpyDeviceToHost, on.s));
  NWG_CUDA_TRY(cudaStreamSynchronize(on.s));
  *same = h == 0;
  return NWG_OK;
}

}  // namespace

// The pieces of a CSR's vertices of more than kHubPiece edges (vertex << 32 |
// piece), in an allocation that the caller frees, also after an error;
// synchronises.
int hub_pieces(const GraphDev* g, const uint64_t* off, uint64_t m, cudaStream_t stream, uint64_t** piece,
               uint64_t* count) {
  const uint64_t cap = 2 * (m / kHubPiece) + 1;  // a vertex of d > kHubPiece edges has at most 2 floor(d / kHubPiece) pieces
  if (cudaMalloc(piece, (cap + 1) * 8) != cudaSuccess) {
    cudaGetLastError();
    *piece = nullptr;
    return set_error(NWG_ENOMEM, "hub list allocation failed (m=" + std::to_string(m) + ")");
  }
  auto* const c = reinterpret_cast<unsigned long long*>(*piece + cap);
  NWG_CUDA_TRY(cudaMemsetAsync(c, 0, 8, stream));
  k_tr_pieces<<<grid_tr(g, g->n, kTrThreads), kTrThreads, 0, stream>>>(off, g->n, *piece, cap, c);
  NWG_CUDA_TRY(cudaGetLastError());
  NWG_CUDA_TRY(cudaMemcpyAsync(count, c, 8, cudaMemcpyDeviceToHost, stream));
  NWG_CUDA_TRY(cudaStreamSynchronize(stream));
  *count = std::min<uint64_t>(*count, cap);
  return NWG_OK;
}

// Whether the in-CSR holds the out-CSR's edges, reversed; compared on a
// graph's first call, on the current device.
int csrs_transposed(GraphDev* g, bool* yes) {
  std::lock_guard<std::mutex> lk(g->transposed_mu);
  if (g->transposed < 0) {
    bool      same = false;
    const int rc   = compare_csrs(g, &same);
    if (rc) return rc;
    g->transposed = same ? 1 : 0;
  }
  *yes = g->transposed == 1;
  return NWG_OK;
}

}  // namespace nwg
