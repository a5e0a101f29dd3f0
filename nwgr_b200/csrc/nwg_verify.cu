// Device BFSVerifier: the checks of nw::graph::BFSVerifier(g, g_t, source,
// parent) (include/nwgraph/algorithms/bfs.hpp:44-98 in NWGraph) on the GPU.
//
//   1. depth = BFS depths from the source over the out-graph (bfs.hpp:47-63).
//      Computed by a plain level-synchronous BFS written only for this check:
//      it shares no code with the direction-optimizing kernels it is used to
//      verify.
//   2. For every vertex u (bfs.hpp:64-96): when depth[u] and parent[u] are
//      both set, the source must be its own parent at depth 0, and any other
//      u must find parent[u] among its in-neighbours (g_t) with
//      depth[parent[u]] == depth[u] - 1; otherwise depth[u] must equal
//      parent[u] (both unset).
//
// The reference stops at the first failing vertex in vertex order; here
// every vertex is checked in parallel and the lowest failing one is kept
// (a 64-bit atomicMin on vertex << 3 | reason), so the verdict, the vertex
// and the reason are the ones the reference reports.
//
// The depths' BFS: a level either pushes from a queue of 64-edge pieces of
// its vertices (so a hub is spread over the grid: with a warp per vertex the
// hub level of RMAT-22 alone took 4.6 of 10.4 ms) or, when its out-edges are
// many, pulls over the visited bitmap.  Depths are defined on the out-graph
// alone, so only a graph whose in-CSR is its out-CSR's transpose pulls
// (csrs_transposed: the traversal under test may rest on the same in-CSR); any
// other pushes every level.  A queue holds n / 4 + m / 512 pieces; a level that
// does not fit is pulled, or its vertices are found by their depths and each is
// pushed by a warp.  No unvisited vertex of a graph that pulls has an
// in-neighbour of an earlier level than the last complete one (that level
// would have visited it), so every visited in-neighbour is one level up; the
// pull reads one copy of the bitmap and writes the other, whose difference
// afterwards is the level.  A level is two launches that read the level's
// counts from device memory (building the queue after a pull; the step), so
// the host enqueues many levels and reads the counts back once.
//
// Bound: gathers of single visited bits and columns (latency); RMAT-22 on a
// B200: 0.5 ms against 10.4 with a warp per frontier vertex and a lane's
// in-edges tested one by one.
#include <algorithm>
#include <cstddef>
#include <string>

#include "nwg_internal.cuh"

using namespace nwg;

#define NWG_API extern "C" __attribute__((visibility("default")))

namespace {

constexpr int      kVThreads = 256;
constexpr uint32_t kUnset    = 0xFFFFFFFFu;  // std::numeric_limits<uint32_t>::max()
constexpr uint32_t kVPiece   = 64;           // out-edges per queue entry: eight lanes, eight edges each
constexpr uint32_t kVProbe   = 8;            // in-edges a lane reads per round
constexpr uint32_t kVLane    = 32;           // in-edges a lane scans alone before the warp helps
constexpr uint32_t kVHub     = 1024;         // a longer rest of a list is checked by the grid, in pieces of this
constexpr uint32_t kVBatch   = 32;           // most levels enqueued before the counts are read back

// One level's frontier, complete when its step runs.
struct VerifyLevel {
  unsigned long long verts;      // vertices of the level
  unsigned long long edges;      // their out-edges
  unsigned long long entries;    // queue entries
  unsigned long long unpushed;   // out-edges of the graph not yet of any level before
  unsigned int       from_pull;  // found by a pull: the queue is not built
  unsigned int       cur;        // which copy of the visited bitmap is current
};

struct VerifyCounters {
  unsigned long long first;    // min over failing vertices of (u << 3 | reason)
  unsigned long long reached;  // vertices with a depth
  unsigned long long pieces;   // pieces of long in-lists
  unsigned long long pad;
  VerifyLevel        lv[kVBatch + 1];
};

struct VerifyArgs {
  const uint64_t* off;
  const uint32_t* col;
  const uint64_t* in_off;
  const uint32_t* in_col;
  uint64_t        n, m;
  uint32_t        use_in;  // the in-CSR is the out-CSR's transpose: levels may pull
  uint32_t*       depth;
  uint32_t*       vis[2];  // visited bitmap, two copies
  uint64_t*       q[2];    // vertex << 32 | piece
  uint64_t        qcap;
  VerifyCounters* cnt;
};

// Pull, where the in-CSR allows it, when the level's out-edges are a good part
// of what is left (and not a handful), or its queue entries did not fit.
__device__ __forceinline__ bool v_pulls(const VerifyArgs& a, const VerifyLevel& l) {
  return a.use_in && (l.entries > a.qcap || (l.edges > l.unpushed / 15 && l.edges > a.n / 32));
}

__global__ void k_v_init(VerifyArgs a, uint32_t source) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t t      = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t deg    = a.off[source + 1] - a.off[source];
  const uint64_t np     = (deg + kVPiece - 1) / kVPiece;
  for (uint64_t i = t; i < a.n; i += stride) a.depth[i] = (i == source) ? 0u : kUnset;
  for (uint64_t w = t; w < (a.n + 31) / 32; w += stride)
    a.vis[0][w] = w == source >> 5 ? 1u << (source & 31) : 0u;
  for (uint64_t i = t; i < np && i < a.qcap; i += stride) a.q[0][i] = ((uint64_t)source << 32) | i;
  if (t == 0) {
    a.cnt->first   = ~0ull;
    a.cnt->reached = 0;
    a.cnt->pieces  = 0;
    a.cnt->lv[0]   = VerifyLevel{1, deg, np, a.m, 0, 0};
  }
}

// Appends the warp's vertices (lane's v where `has`, out-degree deg) to q as
// pieces.  All lanes call.
__device__ __forceinline__ void v_append(const VerifyArgs& a, uint64_t* q, unsigned long long* entries, bool has,
                                         uint32_t v, uint64_t deg) {
  const unsigned     lane = threadIdx.x & 31;
  const uint64_t     np   = has ? (deg + kVPiece - 1) / kVPiece : 0;
  unsigned long long inc  = np;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long x = __shfl_up_sync(kFullMask, inc, o);
    if ((int)lane >= o) inc += x;
  }
  const unsigned long long tot = __shfl_sync(kFullMask, inc, 31);
  if (tot == 0) return;
  unsigned long long base = 0;
  if (lane == 31) base = atomicAdd(entries, tot);
  base                         = __shfl_sync(kFullMask, base, 31);
  const unsigned long long pos = base + inc - np;
  if (np && np <= 8)
    for (uint64_t j = 0; j < np; ++j)
      if (pos + j < a.qcap) q[pos + j] = ((uint64_t)v << 32) | j;
  unsigned big = __ballot_sync(kFullMask, np > 8);
  while (big) {  // the whole warp writes a hub's
    const int src = __ffs(big) - 1;
    big &= big - 1;
    const uint64_t           vs = __shfl_sync(kFullMask, (uint64_t)v, src);
    const unsigned long long ps = __shfl_sync(kFullMask, pos, src);
    const uint64_t           ns = __shfl_sync(kFullMask, np, src);
    for (uint64_t j = lane; j < ns; j += 32)
      if (ps + j < a.qcap) q[ps + j] = (vs << 32) | j;
  }
}

// The queue of level L, when it was found by a pull and will push.
__global__ void __launch_bounds__(kVThreads) k_v_queue(VerifyArgs a, uint32_t L, uint32_t q) {
  VerifyLevel& l = a.cnt->lv[L];
  if (l.verts == 0 || !l.from_pull || v_pulls(a, VerifyLevel{l.verts, l.edges, 0, l.unpushed, 0, 0})) return;
  const uint32_t* cur    = a.vis[l.cur];
  const uint32_t* old    = a.vis[l.cur ^ 1];
  const unsigned  lane   = threadIdx.x & 31;
  const uint64_t  nwords = (a.n + 31) / 32;
  const uint64_t  nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nwords; w += nwarps) {
    const uint32_t d = cur[w] ^ old[w];
    if (!d) continue;
    const bool     has = (d >> lane) & 1u;
    const uint32_t v   = (uint32_t)(w * 32 + lane);
    v_append(a, a.q[q], &l.entries, has, v, has ? a.off[v + 1] - a.off[v] : 0);
  }
}

template <typename T>
__device__ __forceinline__ T v_block_sum(T x) {
  __shared__ T red[kVThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(kFullMask, x, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
  __syncthreads();
  T t = 0;
#pragma unroll
  for (int i = 0; i < kVThreads / 32; ++i) t += red[i];
  return t;
}

// Pushes four edges of the lane (targets x, kUnset = none) of a vertex at
// `level`.  All lanes call.
__device__ __forceinline__ void v_push(const VerifyArgs& a, uint32_t* cur, uint64_t* qo, unsigned long long* entries,
                                       uint32_t level, const uint32_t (&x)[4], unsigned long long& verts,
                                       unsigned long long& edges) {
  bool won[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint32_t bit = 1u << (x[k] & 31);
    // a stale word only costs an atomic: bits go from 0 to 1
    won[k] = x[k] != kUnset && !(cur[x[k] >> 5] & bit) && !(atomicOr(cur + (x[k] >> 5), bit) & bit);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (!__any_sync(kFullMask, won[k])) continue;
    uint64_t deg = 0;
    if (won[k]) {
      a.depth[x[k]] = level + 1;
      deg           = a.off[x[k] + 1] - a.off[x[k]];
      verts += 1;
      edges += deg;
    }
    v_append(a, qo, entries, won[k], x[k], deg);
  }
}

// The step of level L (depth `level`): discoveries get depth level + 1 and
// are counted in lv[L + 1].
__global__ void __launch_bounds__(kVThreads) k_v_step(VerifyArgs a, uint32_t L, uint32_t q, uint32_t level) {
  const VerifyLevel l  = a.cnt->lv[L];
  VerifyLevel&      nl = a.cnt->lv[L + 1];
  if (l.verts == 0) return;
  const bool         pull  = v_pulls(a, l);
  const unsigned     lane  = threadIdx.x & 31;
  const uint64_t     warp  = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t     nwarp = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  unsigned long long verts = 0, edges = 0;
  uint32_t* const    cur   = a.vis[l.cur];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    nl.unpushed  = l.unpushed - min(l.unpushed, l.edges);
    nl.from_pull = pull;
    nl.cur       = l.cur ^ (pull ? 1u : 0u);
  }
  if (pull) {
    uint32_t* const next   = a.vis[l.cur ^ 1];
    const uint64_t  nwords = (a.n + 31) / 32;
    for (uint64_t w = warp; w < nwords; w += nwarp) {
      const uint32_t seen = cur[w];
      const uint32_t u    = (uint32_t)(w * 32 + lane);
      bool           need = u < a.n && !((seen >> lane) & 1u);
      uint64_t       e = 0, end = 0;
      if (need) {
        e    = a.in_off[u];
        end  = a.in_off[u + 1];
        need = e < end;
      }
      bool           found = false;
      const uint64_t lim   = min(end, e + kVLane);
      while (need && e < lim) {
        uint32_t x[kVProbe];
#pragma unroll
        for (uint32_t k = 0; k < kVProbe; ++k) x[k] = e + k < lim ? __ldg(a.in_col + e + k) : kUnset;
#pragma unroll
        for (uint32_t k = 0; k < kVProbe; ++k)
          if (x[k] != kUnset && ((cur[x[k] >> 5] >> (x[k] & 31)) & 1u)) found = true;
        e += kVProbe;
        if (found) need = false;
      }
      unsigned pend = __ballot_sync(kFullMask, need && e < end);
      while (pend) {  // the rest of long lists: the warp together
        const int ld = __ffs(pend) - 1;
        pend &= pend - 1;
        const uint64_t b  = __shfl_sync(kFullMask, e, ld);
        const uint64_t en = __shfl_sync(kFullMask, end, ld);
        bool           hit = false;
        for (uint64_t base = b; base < en && !hit; base += 32 * 4) {
          uint32_t x[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) x[k] = base + k * 32 + lane < en ? __ldg(a.in_col + base + k * 32 + lane) : kUnset;
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (x[k] != kUnset && ((cur[x[k] >> 5] >> (x[k] & 31)) & 1u)) hit = true;
          hit = __any_sync(kFullMask, hit);
        }
        if ((int)lane == ld) found = hit;
      }
      const uint32_t fresh = __ballot_sync(kFullMask, found);
      if (found) {
        a.depth[u] = level + 1;
        verts += 1;
        edges += a.off[u + 1] - a.off[u];
      }
      if (lane == 0) next[w] = seen | fresh;
    }
  } else {
    const uint64_t  count = l.entries > a.qcap ? 0 : l.entries;  // more: k_v_scan's
    const uint64_t* qi    = a.q[q];
    uint64_t* const qo    = a.q[q ^ 1];
    for (uint64_t i0 = warp * 4; i0 < count; i0 += nwarp * 4) {  // four entries per warp, eight lanes each
      const uint64_t i = i0 + (lane >> 3);
      uint64_t       e = 0, end = 0;
      if (i < count) {
        const uint64_t ent = qi[i];
        const uint64_t ob  = a.off[ent >> 32];
        const uint64_t at  = ob + (uint64_t)(uint32_t)ent * kVPiece;
        e                  = at + (lane & 7);
        end                = min(a.off[(ent >> 32) + 1], at + kVPiece);
      }
      while (__any_sync(kFullMask, e < end)) {
        uint32_t x[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) x[k] = e + 8 * k < end ? __ldg(a.col + e + 8 * k) : kUnset;
        v_push(a, cur, qo, &nl.entries, level, x, verts, edges);
        e += 32;
      }
    }
  }
  const unsigned long long vs = v_block_sum(verts), es = v_block_sum(edges);
  if (threadIdx.x == 0 && vs) {
    atomicAdd(&nl.verts, vs);
    atomicAdd(&nl.edges, es);
  }
}

// The pushes of level L where its pieces did not fit the queue, on graphs that
// may not pull: the level's vertices are found by their depths, a warp each.
__global__ void __launch_bounds__(kVThreads) k_v_scan(VerifyArgs a, uint32_t L, uint32_t q, uint32_t level) {
  const VerifyLevel l = a.cnt->lv[L];
  if (l.verts == 0 || l.entries <= a.qcap) return;
  VerifyLevel&       nl    = a.cnt->lv[L + 1];
  uint32_t* const    cur   = a.vis[0];  // only pulls change copies
  const unsigned     lane  = threadIdx.x & 31;
  const uint64_t     nwarp = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  unsigned long long verts = 0, edges = 0;
  for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w * 32 < a.n; w += nwarp) {
    const uint64_t u    = w * 32 + lane;
    unsigned       pend = __ballot_sync(kFullMask, u < a.n && a.depth[u] == level);
    while (pend) {
      const uint64_t us = w * 32 + __ffs(pend) - 1;
      pend &= pend - 1;
      const uint64_t end = a.off[us + 1];
      for (uint64_t e = a.off[us]; e < end; e += 32 * 4) {
        uint32_t x[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) x[k] = e + k * 32 + lane < end ? __ldg(a.col + e + k * 32 + lane) : kUnset;
        v_push(a, cur, a.q[q ^ 1], &nl.entries, level, x, verts, edges);
      }
    }
  }
  const unsigned long long vs = v_block_sum(verts), es = v_block_sum(edges);
  if (threadIdx.x == 0 && vs) {
    atomicAdd(&nl.verts, vs);
    atomicAdd(&nl.edges, es);
  }
}

// The next batch of levels starts from the last one's result.
__global__ void k_v_carry(VerifyCounters* cnt) {
  const VerifyLevel last = cnt->lv[kVBatch];
  __syncthreads();
  for (uint32_t i = threadIdx.x; i <= kVBatch; i += blockDim.x) cnt->lv[i] = i ? VerifyLevel{} : last;
}

__device__ __forceinline__ void v_fail(VerifyCounters* cnt, uint64_t u, uint32_t reason) {
  atomicMin(&cnt->first, ((unsigned long long)u << 3) | reason);
}

// The per-vertex checks (reasons: 1 source wrong, 2 wrong depths, 3 no edge
// from the parent, 4 reachability).  Lanes take consecutive vertices and scan
// up to kVLane in-neighbours alone, kVProbe per round; the warp scans up to
// kVHub more of a longer list; what is left is put down in pieces for
// k_v_pieces.  piece: room for m / kVHub + the number of such lists.
__global__ void __launch_bounds__(kVThreads) k_v_check(VerifyArgs a, const uint32_t* __restrict__ parent,
                                                       uint32_t source, uint64_t* piece) {
  const unsigned     lane    = threadIdx.x & 31;
  const uint64_t     stride  = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t     n_up    = (a.n + 31) & ~31ull;
  unsigned long long reached = 0;
  for (uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; u < n_up; u += stride) {
    const bool     valid = u < a.n;
    const uint32_t du    = valid ? a.depth[u] : kUnset;
    const uint32_t pu    = valid ? parent[u] : kUnset;
    uint32_t       fail  = 0;
    bool           need  = false;  // parent search still open
    uint64_t       e = 0, end = 0;
    if (valid) {
      if (du != kUnset) ++reached;
      if (du != kUnset && pu != kUnset) {
        if (u == source) {
          if (!(pu == u && du == 0)) fail = 1;
        } else {
          e    = a.in_off[u];
          end  = a.in_off[u + 1];
          need = true;
        }
      } else if (du != pu) {
        fail = 4;
      }
    }
    const bool search = need;
    bool       found  = false;
    {
      const uint64_t lim = min(end, e + kVLane);
      while (need && e < lim) {
#pragma unroll
        for (uint32_t k = 0; k < kVProbe; ++k)
          if (e + k < lim && __ldg(a.in_col + e + k) == pu) found = true;
        e = min(lim, e + kVProbe);
        if (found) need = false;
      }
    }
    unsigned pend = __ballot_sync(kFullMask, need && e < end);
    bool     open = false;  // the grid scans the rest
    while (pend) {
      const int ld = __ffs(pend) - 1;
      pend &= pend - 1;
      const uint64_t b   = __shfl_sync(kFullMask, e, ld);
      const uint64_t en  = __shfl_sync(kFullMask, end, ld);
      const uint32_t pp  = __shfl_sync(kFullMask, pu, ld);
      const uint64_t lim = min(en, b + kVHub);
      bool           hit = false;
      for (uint64_t base = b; base < lim && !hit; base += 32 * kVProbe) {
#pragma unroll
        for (uint32_t k = 0; k < kVProbe; ++k) {
          const uint64_t i = base + k * 32 + lane;
          if (i < lim && __ldg(a.in_col + i) == pp) hit = true;
        }
        hit = __any_sync(kFullMask, hit);
      }
      if (!hit && lim < en) {
        const uint64_t     np = (en - lim + kVHub - 1) / kVHub;
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(&a.cnt->pieces, (unsigned long long)np);
        at                = __shfl_sync(kFullMask, at, 0);
        const uint64_t us = __shfl_sync(kFullMask, u, ld);
        for (uint64_t j = lane; j < np; j += 32) piece[at + j] = (us << 32) | j;
        if ((int)lane == ld) open = true;
      }
      if ((int)lane == ld) found = hit;
    }
    if (search && !open) {
      if (!found) fail = 3;
      else if (du == 0 || a.depth[pu] != du - 1) fail = 2;  // the parent's depth (bfs.hpp:79)
    }
    if (fail) v_fail(a.cnt, u, fail);
  }
  const unsigned long long r = v_block_sum(reached);
  if (threadIdx.x == 0 && r) atomicAdd(&a.cnt->reached, r);
}

// A warp per piece of a long in-list: a hit sets the vertex's bit in
// `found` (all zero before).
__global__ void __launch_bounds__(kVThreads) k_v_pieces(VerifyArgs a, const uint32_t* __restrict__ parent,
                                                        const uint64_t* __restrict__ piece, uint32_t* found) {
  const unsigned lane   = threadIdx.x & 31;
  const uint64_t count  = a.cnt->pieces;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < count; i += nwarps) {
    const uint64_t u   = piece[i] >> 32;
    const uint64_t en  = a.in_off[u + 1];
    const uint64_t b   = a.in_off[u] + kVLane + kVHub + (piece[i] & 0xFFFFFFFFull) * kVHub;
    const uint64_t lim = min(en, b + kVHub);
    const uint32_t pp  = parent[u];
    bool           hit = false;
    for (uint64_t base = b; base < lim && !hit; base += 32 * kVProbe) {
#pragma unroll
      for (uint32_t k = 0; k < kVProbe; ++k) {
        const uint64_t j = base + k * 32 + lane;
        if (j < lim && __ldg(a.in_col + j) == pp) hit = true;
      }
      hit = __any_sync(kFullMask, hit);
    }
    if (hit && lane == 0) atomicOr(found + (u >> 5), 1u << (u & 31));
  }
}

// The verdict of every vertex that was put down in pieces.
__global__ void k_v_verdicts(VerifyArgs a, const uint32_t* __restrict__ parent, const uint64_t* __restrict__ piece,
                             const uint32_t* __restrict__ found) {
  const uint64_t count = a.cnt->pieces;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (uint64_t)gridDim.x * blockDim.x) {
    if (piece[i] & 0xFFFFFFFFull) continue;
    const uint64_t u  = piece[i] >> 32;
    const uint32_t du = a.depth[u];
    if (!((found[u >> 5] >> (u & 31)) & 1u)) v_fail(a.cnt, u, 3);
    else if (du == 0 || a.depth[parent[u]] != du - 1) v_fail(a.cnt, u, 2);
  }
}

int grid_v(const GraphDev* g, uint64_t items, uint64_t per_block) {
  const uint64_t want = (items + per_block - 1) / per_block;
  return (int)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)g->sm_count * 8, want));
}

}  // namespace

namespace nwg {

// The check's state, made on a graph's first verification and kept with it
// (making and freeing it took 2 ms of a call); a call beside another on the
// same graph makes its own.
// The counters are read through a slot of the process's pinned memory: with a
// pinned mirror of its own a first verification of a graph of 1,024 vertices
// took 2.0-4.0 ms, 0.26 so; read into ordinary memory, a call over 40
// levels took 4% longer.  One allocation for all arrays made a uniform graph of
// 2^24 vertices 3% slower (12.5 ms against 12.9).
struct VerifyWs {
  int             device     = 0;
  uint64_t        kept_bytes = 0;
  bool            ready   = false;
  bool            use_in  = false;    // csrs_transposed
  VerifyCounters* cnt     = nullptr;
  uint32_t*       depth   = nullptr;
  uint32_t*       vis     = nullptr;  // both copies
  uint64_t*       q       = nullptr;  // both queues; the pieces of long in-lists after the traversal
  uint32_t*       par     = nullptr;  // device copy of host parents, made when first needed
  cudaStream_t    s       = nullptr;
  cudaEvent_t     ev0 = nullptr, ev1 = nullptr;
};

void verify_ws_free(VerifyWs* b) {
  if (!b) return;
  drop_bytes(b->device, b->kept_bytes);
  if (b->s) cudaStreamSynchronize(b->s);
  cudaFree(b->depth);
  cudaFree(b->vis);
  cudaFree(b->q);
  cudaFree(b->cnt);
  cudaFree(b->par);
  if (b->ev0) cudaEventDestroy(b->ev0);
  if (b->ev1) cudaEventDestroy(b->ev1);
  if (b->s) cudaStreamDestroy(b->s);
  delete b;
}

}  // namespace nwg

namespace {

uint64_t queue_cap(const GraphDev* g) { return g->n / 4 + g->m / 512 + 1; }

// Both queues, whose memory takes the pieces of long in-lists afterwards: in_m
// / kVHub entries plus one per list of over kVHub, at most twice that.
uint64_t queue_words(const GraphDev* g) {
  return std::max<uint64_t>(2 * queue_cap(g), 2 * (g->in_m / kVHub) + 2);
}

int verify_ws_make(GraphDev* g, VerifyWs& b) {
  if (!b.s) NWG_CUDA_TRY(cudaStreamCreateWithFlags(&b.s, cudaStreamNonBlocking));
  const int rc = csrs_transposed(g, b.s, &b.use_in);
  if (rc) return rc;
  if ((!b.depth && cudaMalloc(&b.depth, g->n * 4) != cudaSuccess) ||
      (!b.vis && cudaMalloc(&b.vis, 2 * ((g->n + 31) / 32) * 4) != cudaSuccess) ||
      (!b.q && cudaMalloc(&b.q, queue_words(g) * 8) != cudaSuccess) ||
      (!b.cnt && cudaMalloc(&b.cnt, sizeof(VerifyCounters)) != cudaSuccess)) {
    cudaGetLastError();
    return set_error(NWG_ENOMEM, "verifier allocation failed (n=" + std::to_string(g->n) + ")");
  }
  if (!b.ev0) NWG_CUDA_TRY(cudaEventCreate(&b.ev0));
  if (!b.ev1) NWG_CUDA_TRY(cudaEventCreate(&b.ev1));
  b.ready = true;
  return NWG_OK;
}

int verify_on(GraphDev* g, VerifyWs& b, uint32_t source, const uint32_t* parents_host, const uint32_t* parents_dev,
              nwg_verify_result* out) {
  const uint64_t n = g->n;
  if (!b.ready) {
    const int rc = verify_ws_make(g, b);
    if (rc) return rc;
  }
  if (parents_host && !b.par && cudaMalloc(&b.par, std::max<uint64_t>(n, 1) * 4) != cudaSuccess) {
    cudaGetLastError();
    b.par = nullptr;
    return set_error(NWG_ENOMEM, "verifier allocation failed (n=" + std::to_string(n) + ")");
  }
  VerifyArgs a;
  a.off    = g->off;
  a.col    = g->col;
  a.in_off = g->in_off;
  a.in_col = g->in_col;
  a.n      = n;
  a.m      = g->m;
  a.use_in = b.use_in ? 1u : 0u;
  a.depth  = b.depth;
  a.vis[0] = b.vis;
  a.vis[1] = b.vis + (n + 31) / 32;
  a.q[0]   = b.q;
  a.qcap   = queue_cap(g);
  a.q[1]   = b.q + a.qcap;
  a.cnt    = b.cnt;
  NWG_CUDA_TRY(cudaEventRecord(b.ev0, b.s));
  const uint32_t* par = parents_dev;
  if (parents_host) {
    NWG_CUDA_TRY(cudaMemcpyAsync(b.par, parents_host, n * 4, cudaMemcpyHostToDevice, b.s));
    par = b.par;
  }
  NWG_CUDA_TRY(cudaMemsetAsync(b.cnt, 0, sizeof(VerifyCounters), b.s));
  k_v_init<<<grid_v(g, n, kVThreads), kVThreads, 0, b.s>>>(a, source);
  const int gw = grid_v(g, std::max(n, g->m / kVPiece), kVThreads);  // a step's grid: levels of any size
  uint32_t  base = 0;  // depth of the batch's first level, lv[0]
  uint32_t  levels = 0;
  PinnedSlot      slot;
  VerifyCounters& hc = *slot.as<VerifyCounters>();
  // the first read-back after eight levels (hub graphs have 5-9), then every kVBatch
  for (uint32_t done = 0, until = 8;;) {
    for (; done < until; ++done) {
      const uint32_t level = base + done;
      k_v_queue<<<gw, kVThreads, 0, b.s>>>(a, done, level & 1);
      if (!b.use_in) k_v_scan<<<gw, kVThreads, 0, b.s>>>(a, done, level & 1, level);
      k_v_step<<<gw, kVThreads, 0, b.s>>>(a, done, level & 1, level);
    }
    NWG_CUDA_TRY(cudaGetLastError());
    NWG_CUDA_TRY(cudaMemcpyAsync(&hc, b.cnt, sizeof hc, cudaMemcpyDeviceToHost, b.s));
    NWG_CUDA_TRY(cudaStreamSynchronize(b.s));
    if (hc.lv[done].verts == 0) {
      while (hc.lv[done].verts == 0) --done;  // lv[0] holds a vertex
      levels = base + done + 1;
      break;
    }
    if (done == kVBatch) {
      k_v_carry<<<1, 64, 0, b.s>>>(b.cnt);
      base += kVBatch;
      done = 0;
    }
    until = kVBatch;
  }
  // found bits of the long lists: the first bitmap copy, free now
  const uint64_t words = (n + 31) / 32;
  NWG_CUDA_TRY(cudaMemsetAsync(b.vis, 0, words * 4, b.s));
  k_v_check<<<grid_v(g, n, kVThreads), kVThreads, 0, b.s>>>(a, par, source, b.q);
  k_v_pieces<<<grid_v(g, g->in_m / kVHub, kVThreads / 32), kVThreads, 0, b.s>>>(a, par, b.q, b.vis);
  k_v_verdicts<<<grid_v(g, g->in_m / kVHub, kVThreads), kVThreads, 0, b.s>>>(a, par, b.q, b.vis);
  NWG_CUDA_TRY(cudaGetLastError());
  NWG_CUDA_TRY(cudaEventRecord(b.ev1, b.s));
  NWG_CUDA_TRY(cudaMemcpyAsync(&hc, b.cnt, offsetof(VerifyCounters, lv), cudaMemcpyDeviceToHost, b.s));
  NWG_CUDA_TRY(cudaStreamSynchronize(b.s));
  nwg_verify_result r = {};
  r.valid             = hc.first == ~0ull ? 1 : 0;
  r.reason            = r.valid ? 0u : (uint32_t)(hc.first & 7u);
  r.first_bad         = r.valid ? ~0ull : (hc.first >> 3);
  r.reached           = hc.reached;
  r.levels            = levels;
  cudaEventElapsedTime(&r.device_ms, b.ev0, b.ev1);
  *out = r;
  return NWG_OK;
}

int verify(GraphDev* g, uint32_t source, const uint32_t* parents_host, const uint32_t* parents_dev,
           nwg_verify_result* out) {
  KeptState<VerifyWs, verify_ws_free> b(g->kept_mu, g->verify_ws);
  const int rc = verify_on(g, *b, source, parents_host, parents_dev, out);
  if (!rc) b.keep(g->device, 4 * g->n * (b->par ? 2 : 1) + g->n / 4 + queue_words(g) * 8);
  return rc;
}

}  // namespace

NWG_API int nwg_verify(nwg_graph h, uint32_t source, const uint32_t* parents_host, const uint32_t* parents_dev,
                       nwg_verify_result* result) {
  try {
    if (!h || !result || (!parents_host == !parents_dev))
      return set_error(NWG_EINVAL, "NULL graph or result, or not exactly one of parents_host / parents_dev");
    auto* g = reinterpret_cast<GraphDev*>(h);
    if (source >= g->n) return set_error(NWG_EINVAL, "source " + std::to_string(source) + " >= n");
    int prev = 0;
    cudaGetDevice(&prev);
    if (prev != g->device) cudaSetDevice(g->device);
    const int rc = verify(g, source, parents_host, parents_dev, result);
    if (prev != g->device) cudaSetDevice(prev);
    return rc;
  } catch (const std::exception& ex) {
    return set_error(NWG_ENOMEM, std::string("verifier failed: ") + ex.what());
  }
}
