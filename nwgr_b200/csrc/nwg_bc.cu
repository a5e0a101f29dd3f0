// Approximate betweenness centrality over a list of sources (Brandes), the
// computation of NWGraph's brandes_bc<float, double>(graph, sources, threads,
// ..., normalize) (include/nwgraph/algorithms/betweenness_centrality.hpp:
// 218-324 in NWGraph), on the GPU.
//
// Per source, over the out-graph:
//   forward  -- level-synchronous BFS from the source; every edge u -> v with
//               level[v] == level[u] + 1 adds path_counts[u] to
//               path_counts[v] (double; the reference's accum_t).  That edge
//               test is the reference's succ bit (set when v is new or on
//               the level being built, :262-266), recomputed instead of
//               stored.
//   backward -- levels deepest first: delta[u] = sum over those edges of
//               path_counts[u] / path_counts[v] * (1 + delta[v]), and
//               bc[u] += delta[u] for every reached vertex, the source
//               included (:297-307).
// Then bc /= max(bc) when normalizing (:316-319).
//
// Forward, a level either pushes (the vertices of the level add their path
// counts to their new out-neighbours: levels claimed with atomicCAS, counts
// added with double atomics) or, when its out-edges are many against the
// in-edges of what is left, pulls: every unvisited vertex sums the path
// counts of its visited in-neighbours, without an atomic.  All of those are
// one level up, since a vertex with an in-neighbour further up would have
// been visited by the level after it.  The pull tests a bit of the visited
// bitmap (128 KB at 2^20 vertices) before it reads a count; it reads one
// copy of the bitmap and writes the other.  Path counts are integers: exact
// below 2^53, so the order of the adds does not matter.  On RMAT-20 the hub
// level took 0.88 ms as a push (contended double atomics) and the level
// after it 0.34 ms for a few discoveries.
//
// Backward, a level sums its terms from its own out-edges or, when the level
// below has far fewer in-edges, is added to by that level; the first needs
// no atomics except for hubs.
//
// Pulls and scatters read the in-CSR.  The computation itself is defined on
// the out-graph alone, and a graph registered without an in-CSR may in fact
// be directed, so the graph's two CSRs are compared (csrs_transposed); where
// they differ every level pushes and gathers.
//
// Work split: eight lanes per vertex; vertices of more than kBcHub edges in
// pieces of that many, a warp each, from a list made once per graph (a
// level's hubs are found in it by their level).  Forward levels are enqueued
// without a read-back between them (a step reads the level's counts from
// device memory); the host reads them every few levels.
//
// Every vertex's level, dependency and path count (or, once its dependency
// is final, its weight) share one 16-byte record.  Several sources run at
// once, one host thread and stream each.  Scores are float sums across
// sources, as in the reference.
#include <algorithm>
#include <atomic>
#include <string>
#include <thread>
#include <vector>

#include "nwg_internal.cuh"

using namespace nwg;

#define NWG_API extern "C" __attribute__((visibility("default")))

namespace {

constexpr int      kBcThreads = 256;
constexpr uint32_t kBcHub     = 512;  // a vertex of more edges is split into pieces of this many
constexpr uint32_t kBcBatch   = 32;   // most forward levels enqueued before a read-back
constexpr uint32_t kUnset     = 0xFFFFFFFFu;

// Per-vertex state of one source, one 16-byte record so that a backward
// edge reads its target's level, dependency and path count in one sector.
struct alignas(16) BcVertex {
  uint32_t level;  // BFS level (kUnset = unreached)
  float    delta;  // dependency (score_t)
  double   sigma;  // shortest-path count (accum_t), or the weight (1 + delta) / count
};

// A forward level, complete when its step runs.
struct BcLevel {
  unsigned long long verts;   // vertices: order[first, first + verts)
  unsigned long long out;     // their out-edges
  unsigned long long in;      // their in-edges
  unsigned long long first;
  unsigned long long in_rem;  // in-edges of the vertices of no level before this one
  unsigned int       cur;     // which copy of the visited bitmap is current
  unsigned int       pad;
};

struct BcArgs {
  const uint64_t* off;
  const uint32_t* col;
  const uint64_t* in_off;
  const uint32_t* in_col;
  uint64_t        n, m;
  uint32_t        use_in;  // the in-CSR is the out-CSR's transpose: pulls and scatters may read it
  BcVertex*       vx;
  double*         dsum;   // sums of the weights below (zero between uses)
  uint32_t*       order;  // vertices by level
  uint32_t*       vis[2];
  BcLevel*        lv;     // [kBcBatch + 1]
  const uint64_t* piece;  // vertex << 32 | piece of every vertex of more than kBcHub out-edges
  const uint64_t* in_piece;
  uint64_t        npiece, nin_piece;
  float*          bc;
};

// Pull when the level's out-edges are more than a third of the in-edges of
// what is not visited yet, and not a handful: a pushed edge costs about
// three pulled ones (level gather, claim or double atomic add).
__device__ __forceinline__ bool bc_pulls(const BcArgs& a, const BcLevel& l) {
  return a.use_in && l.out > (l.in_rem - min(l.in_rem, l.in)) / 3 && l.out > a.n / 8;
}

// The sums a step's blocks add to the next level.
struct BcSums {
  unsigned long long verts, out, in;
};

__device__ __forceinline__ unsigned long long bc_block_sum(unsigned long long x) {
  __shared__ unsigned long long red[kBcThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(kFullMask, x, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
  __syncthreads();
  unsigned long long t = 0;
#pragma unroll
  for (int i = 0; i < kBcThreads / 32; ++i) t += red[i];
  return t;
}

// The warp's new vertices (lane's v where `has`) to the order, one counter
// update per warp, and their degrees to the sums.  All lanes call.
__device__ __forceinline__ void bc_append(const BcArgs& a, BcLevel& nl, uint64_t first, bool has, uint32_t v,
                                          BcSums& s) {
  const unsigned m = __ballot_sync(kFullMask, has);
  if (!m) return;
  const unsigned     lane = threadIdx.x & 31;
  unsigned long long base = 0;
  if (lane == 0) base = atomicAdd(&nl.verts, (unsigned long long)__popc(m));
  base = __shfl_sync(kFullMask, base, 0);
  if (has) {
    const uint64_t at = first + base + __popc(m & ((1u << lane) - 1u));
    if (at < a.n) a.order[at] = v;  // every vertex is claimed once
    const uint64_t d = a.off[v + 1] - a.off[v];
    s.out += d;
    s.in += a.in_off == a.off ? d : a.in_off[v + 1] - a.in_off[v];
  }
}

// One pushed edge: claim v for level lvl + 1 and add su to its path count.
__device__ __forceinline__ bool bc_push_edge(const BcArgs& a, uint32_t* cur, uint32_t v, double su, uint32_t lvl) {
  bool     won = false;
  uint32_t lv  = a.vx[v].level;
  if (lv == kUnset) {
    lv  = atomicCAS(&a.vx[v].level, kUnset, lvl + 1);
    won = lv == kUnset;
    if (won) {
      lv = lvl + 1;
      atomicOr(cur + (v >> 5), 1u << (v & 31));
    }
  }
  if (lv == lvl + 1) atomicAdd(&a.vx[v].sigma, su);
  return won;
}

// The forward step of level L (BFS level lvl).
__global__ void __launch_bounds__(kBcThreads) k_bc_forward(BcArgs a, uint32_t L, uint32_t lvl) {
  const BcLevel l  = a.lv[L];
  BcLevel&      nl = a.lv[L + 1];
  if (l.verts == 0) return;
  const bool      pull  = bc_pulls(a, l);
  const unsigned  lane  = threadIdx.x & 31;
  const uint64_t  warp  = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t  nwarp = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint64_t  first = l.first + l.verts;
  uint32_t* const cur   = a.vis[l.cur];
  BcSums          s     = {0, 0, 0};
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    nl.first  = first;
    nl.in_rem = l.in_rem - min(l.in_rem, l.in);
    nl.cur    = l.cur ^ (pull ? 1u : 0u);
  }
  if (pull) {
    uint32_t* const next   = a.vis[l.cur ^ 1];  // holds a subset of cur
    const uint64_t  nwords = (a.n + 31) / 32;
    for (uint64_t w = warp; w < nwords; w += nwarp) {
      const uint32_t seen = cur[w];
      const uint32_t u    = (uint32_t)(w * 32 + lane);
      uint64_t       e = 0, end = 0;
      if (u < a.n && !((seen >> lane) & 1u)) {
        e   = a.in_off[u];
        end = a.in_off[u + 1];
        if (end - e > kBcHub) e = end;  // a hub: in pieces below
      }
      double         sum   = 0.0;
      bool           found = false;
      const uint64_t lim   = min(end, e + 32);
      for (; e < lim; e += 8) {
        uint32_t x[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = e + k < lim ? __ldg(a.in_col + e + k) : kUnset;
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (x[k] != kUnset && ((cur[x[k] >> 5] >> (x[k] & 31)) & 1u)) {
            sum += a.vx[x[k]].sigma;
            found = true;
          }
      }
      e             = lim;
      unsigned pend = __ballot_sync(kFullMask, e < end);
      while (pend) {  // the rest of longer lists: the warp together
        const int ld = __ffs(pend) - 1;
        pend &= pend - 1;
        const uint64_t b  = __shfl_sync(kFullMask, e, ld);
        const uint64_t en = __shfl_sync(kFullMask, end, ld);
        double         ps = 0.0;
        bool           pf = false;
        for (uint64_t i0 = b; i0 < en; i0 += 128) {
          uint32_t x[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint64_t i = i0 + k * 32 + lane;
            x[k]             = i < en ? __ldg(a.in_col + i) : kUnset;
          }
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (x[k] != kUnset && ((cur[x[k] >> 5] >> (x[k] & 31)) & 1u)) {
              ps += a.vx[x[k]].sigma;
              pf = true;
            }
        }
        pf = __any_sync(kFullMask, pf);
        if (pf) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) ps += __shfl_xor_sync(kFullMask, ps, o);
          if ((int)lane == ld) {
            sum += ps;
            found = true;
          }
        }
      }
      const uint32_t fresh = __ballot_sync(kFullMask, found);
      if (found) a.vx[u] = BcVertex{lvl + 1, 0.0f, sum};
      if (lane == 0) atomicOr(next + w, seen | fresh);  // a hub's bit may be set meanwhile
      bc_append(a, nl, first, found, u, s);
    }
    for (uint64_t i = warp; i < a.nin_piece; i += nwarp) {
      const uint32_t u = (uint32_t)(a.in_piece[i] >> 32);
      if ((cur[u >> 5] >> (u & 31)) & 1u) continue;  // warp-uniform
      const uint64_t b  = a.in_off[u] + (uint64_t)(uint32_t)a.in_piece[i] * kBcHub;
      const uint64_t en = min(a.in_off[u + 1], b + kBcHub);
      double         ps = 0.0;
      bool           pf = false;
      for (uint64_t i0 = b; i0 < en; i0 += 128) {
        uint32_t x[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint64_t j = i0 + k * 32 + lane;
          x[k]             = j < en ? __ldg(a.in_col + j) : kUnset;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (x[k] != kUnset && ((cur[x[k] >> 5] >> (x[k] & 31)) & 1u)) {
            ps += a.vx[x[k]].sigma;
            pf = true;
          }
      }
      bool won = false;
      if (__any_sync(kFullMask, pf)) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ps += __shfl_xor_sync(kFullMask, ps, o);
        if (lane == 0) {
          atomicAdd(&a.vx[u].sigma, ps);
          won = atomicCAS(&a.vx[u].level, kUnset, lvl + 1) == kUnset;
          if (won) atomicOr(next + (u >> 5), 1u << (u & 31));
        }
      }
      bc_append(a, nl, first, won, u, s);
    }
  } else {
    for (uint64_t i0 = warp * 4; i0 < l.verts; i0 += nwarp * 4) {  // four vertices per warp
      const uint64_t i = i0 + (lane >> 3);
      uint64_t       e = 0, end = 0;
      double         su = 0.0;
      if (i < l.verts) {
        const uint32_t u = a.order[l.first + i];
        su               = a.vx[u].sigma;
        e                = a.off[u];
        end              = a.off[u + 1];
        if (end - e > kBcHub) e = end;  // a hub: in pieces below
        e += lane & 7;
      }
      while (__any_sync(kFullMask, e < end)) {
        uint32_t x[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) x[k] = e + 8 * k < end ? __ldg(a.col + e + 8 * k) : kUnset;
        bool won[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) won[k] = x[k] != kUnset && bc_push_edge(a, cur, x[k], su, lvl);
#pragma unroll
        for (int k = 0; k < 4; ++k) bc_append(a, nl, first, won[k], x[k], s);
        e += 32;
      }
    }
    for (uint64_t i = warp; i < a.npiece; i += nwarp) {
      const uint32_t u = (uint32_t)(a.piece[i] >> 32);
      const BcVertex r = a.vx[u];
      if (r.level != lvl) continue;  // warp-uniform: level lvl is complete, and no other level takes this value now
      const uint64_t b  = a.off[u] + (uint64_t)(uint32_t)a.piece[i] * kBcHub;
      const uint64_t en = min(a.off[u + 1], b + kBcHub);
      for (uint64_t i0 = b; i0 < en; i0 += 128) {
        uint32_t x[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint64_t j = i0 + k * 32 + lane;
          x[k]             = j < en ? __ldg(a.col + j) : kUnset;
        }
        bool won[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) won[k] = x[k] != kUnset && bc_push_edge(a, cur, x[k], r.sigma, lvl);
#pragma unroll
        for (int k = 0; k < 4; ++k) bc_append(a, nl, first, won[k], x[k], s);
      }
    }
  }
  const unsigned long long so = bc_block_sum(s.out), si = bc_block_sum(s.in);
  if (threadIdx.x == 0 && (so | si)) {
    atomicAdd(&nl.out, so);
    atomicAdd(&nl.in, si);
  }
}

// The next batch of levels starts from the last one's result.
__global__ void k_bc_carry(BcLevel* lv) {
  const BcLevel last = lv[kBcBatch];
  __syncthreads();
  for (uint32_t i = threadIdx.x; i <= kBcBatch; i += blockDim.x) lv[i] = i ? BcLevel{} : last;
}

// A vertex's dependency d is final: its score takes it, and as its path
// count is not needed any more its slot takes the weight (1 + d) / count
// that the level above multiplies by: the reference's path_counts[w] /
// path_counts[u] * (1.0f + deltas[u]) (:301) with the division done once per
// vertex instead of once per edge.
//
// The count su multiplies the sum of the weights once, not each of them.  That
// differs in one case: no successors and a count past the range of doubles,
// where inf * 0 would be a NaN that spreads to every vertex above (with
// successors it is NaN in the reference too: their counts are infinite as
// well, their weights 0).  A sum of no terms is therefore kBcNone, -0.0, which
// adding any weight, +0.0 too, changes.  (A product in every term made RMAT-20's
// 8 sources 4.0 ms, 3.4 without.)
constexpr double kBcNone = -0.0;

__device__ __forceinline__ void bc_final(const BcArgs& a, uint32_t u, double su, double sum) {
  const float d = __double_as_longlong(sum) == __double_as_longlong(kBcNone) ? 0.0f : (float)(su * sum);
  a.vx[u].delta = d;
  a.vx[u].sigma = (double)(1.0f + d) / su;
  if (d != 0.0f) atomicAdd(&a.bc[u], d);
}

// Backward by gathering: the sums of order[first, first + count)'s weights
// below (level lvl + 1), each vertex's dependency final at once; hubs add
// their pieces' sums to dsum for k_bc_finish.
__global__ void __launch_bounds__(kBcThreads) k_bc_gather(BcArgs a, uint64_t first, uint64_t count, uint32_t lvl) {
  const unsigned lane  = threadIdx.x & 31;
  const uint64_t warp  = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarp = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t i0 = warp * 4; i0 < count; i0 += nwarp * 4) {
    const uint64_t i = i0 + (lane >> 3);
    uint32_t       u = 0;
    uint64_t       e = 0, end = 0;
    bool           mine = false;
    if (i < count) {
      u    = a.order[first + i];
      e    = a.off[u];
      end  = a.off[u + 1];
      mine = end - e <= kBcHub;
      if (!mine) e = end;
      e += lane & 7;
    }
    double acc = kBcNone;
    for (; e < end; e += 32) {
      uint32_t x[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) x[k] = e + 8 * k < end ? __ldg(a.col + e + 8 * k) : kUnset;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (x[k] != kUnset) {
          const BcVertex r = a.vx[x[k]];  // level and weight in one 16-byte load
          if (r.level == lvl + 1) acc += r.sigma;
        }
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) acc += __shfl_xor_sync(kFullMask, acc, o);
    if (mine && (lane & 7) == 0) bc_final(a, u, a.vx[u].sigma, acc);
  }
  for (uint64_t i = warp; i < a.npiece; i += nwarp) {
    const uint32_t u = (uint32_t)(a.piece[i] >> 32);
    if (a.vx[u].level != lvl) continue;
    const uint64_t b  = a.off[u] + (uint64_t)(uint32_t)a.piece[i] * kBcHub;
    const uint64_t en = min(a.off[u + 1], b + kBcHub);
    double         acc = 0.0;
    for (uint64_t i0 = b; i0 < en; i0 += 128) {
      uint32_t x[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint64_t j = i0 + k * 32 + lane;
        x[k]             = j < en ? __ldg(a.col + j) : kUnset;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (x[k] != kUnset) {
          const BcVertex r = a.vx[x[k]];
          if (r.level == lvl + 1) acc += r.sigma;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(kFullMask, acc, o);
    if (lane == 0 && acc != 0.0) atomicAdd(&a.dsum[u], acc);
  }
}

// Backward by scattering: order[first, first + count) (level lvl + 1) adds
// its weights to its in-neighbours of level lvl; k_bc_finish follows.
__global__ void __launch_bounds__(kBcThreads) k_bc_scatter(BcArgs a, uint64_t first, uint64_t count, uint32_t lvl) {
  const unsigned lane  = threadIdx.x & 31;
  const uint64_t warp  = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarp = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t i0 = warp * 4; i0 < count; i0 += nwarp * 4) {
    const uint64_t i = i0 + (lane >> 3);
    if (i >= count) continue;
    const uint32_t v   = a.order[first + i];
    const uint64_t e   = a.in_off[v], end = a.in_off[v + 1];
    const double   wgt = a.vx[v].sigma;
    if (end - e > kBcHub) continue;
    for (uint64_t j = e + (lane & 7); j < end; j += 8) {
      const uint32_t u = __ldg(a.in_col + j);
      if (a.vx[u].level == lvl) atomicAdd(&a.dsum[u], wgt);
    }
  }
  for (uint64_t i = warp; i < a.nin_piece; i += nwarp) {
    const uint32_t v = (uint32_t)(a.in_piece[i] >> 32);
    const BcVertex r = a.vx[v];
    if (r.level != lvl + 1) continue;
    const uint64_t b  = a.in_off[v] + (uint64_t)(uint32_t)a.in_piece[i] * kBcHub;
    const uint64_t en = min(a.in_off[v + 1], b + kBcHub);
    for (uint64_t j = b + lane; j < en; j += 32) {
      const uint32_t u = __ldg(a.in_col + j);
      if (a.vx[u].level == lvl) atomicAdd(&a.dsum[u], r.sigma);
    }
  }
}

// Whether u, at level lvl, has an out-neighbour at the next one.
__device__ __noinline__ bool bc_has_successor(const uint64_t* off, const uint32_t* col, const BcVertex* vx,
                                              uint32_t u, uint32_t lvl) {
  for (uint64_t e = off[u]; e < off[u + 1]; ++e)
    if (vx[col[e]].level == lvl + 1) return true;
  return false;
}

// The dependencies of order[first, first + count) from dsum, which is zero
// again afterwards; hubs_only after a gather.  dsum does not tell no term from
// terms of 0, which only matters to an infinite count.
__global__ void k_bc_finish(BcArgs a, uint64_t first, uint64_t count, uint32_t hubs_only) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += stride) {
    const uint32_t u = a.order[first + i];
    if (hubs_only && a.off[u + 1] - a.off[u] <= kBcHub) continue;
    const double su  = a.vx[u].sigma;
    double       sum = a.dsum[u];
    if (sum != 0.0) a.dsum[u] = 0.0;
    else if (isinf(su) && !bc_has_successor(a.off, a.col, a.vx, u, a.vx[u].level)) sum = kBcNone;
    bc_final(a, u, su, sum);
  }
}

// Every vertex unreached, no path, no dependency; then the source.
__global__ void k_bc_reset(BcArgs a, uint32_t s) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t t      = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (uint64_t i = t; i < a.n; i += stride)
    a.vx[i] = (i == s) ? BcVertex{0u, 0.0f, 1.0} : BcVertex{kUnset, 0.0f, 0.0};
  for (uint64_t w = t; w < (a.n + 31) / 32; w += stride) {
    const uint32_t b = w == s >> 5 ? 1u << (s & 31) : 0u;
    a.vis[0][w] = a.vis[1][w] = b;
  }
  if (t <= kBcBatch) {
    BcLevel l = {};
    if (t == 0) l = BcLevel{1, a.off[s + 1] - a.off[s], a.in_off[s + 1] - a.in_off[s], 0, a.m, 0, 0};
    a.lv[t] = l;
  }
  if (t == 0) a.order[0] = s;
}

// The pieces of every vertex of more than kBcHub edges.
__global__ void k_bc_pieces(const uint64_t* __restrict__ off, uint64_t n, uint64_t* piece, uint64_t cap,
                            unsigned long long* count) {
  const unsigned lane  = threadIdx.x & 31;
  const uint64_t nwarp = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < (n + 31) / 32; w += nwarp) {
    const uint64_t v    = w * 32 + lane;
    const uint64_t d    = v < n ? off[v + 1] - off[v] : 0;
    unsigned       hubs = __ballot_sync(kFullMask, d > kBcHub);
    while (hubs) {
      const int src = __ffs(hubs) - 1;
      hubs &= hubs - 1;
      const uint64_t     np   = (__shfl_sync(kFullMask, d, src) + kBcHub - 1) / kBcHub;
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(count, (unsigned long long)np);
      base = __shfl_sync(kFullMask, base, 0);
      for (uint64_t j = lane; j < np; j += 32)
        if (base + j < cap) piece[base + j] = ((w * 32 + src) << 32) | j;
    }
  }
}

// Largest score (non-negative floats: their bit patterns order as integers).
__global__ void k_bc_max(const float* bc, uint64_t n, unsigned int* maxbits) {
  unsigned int   m      = 0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    m = max(m, __float_as_uint(fmaxf(bc[i], 0.0f)));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(kFullMask, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(maxbits, m);
}

__global__ void k_bc_divide(float* bc, uint64_t n, const unsigned int* maxbits) {
  const float    big    = __uint_as_float(*maxbits);
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) bc[i] = bc[i] / big;
}

// Grid of a grid-stride kernel: no more blocks than fit on the GPU at once
// (the tasks are dealt out statically, so blocks of a second wave would
// start only when the first wave ends), and no more than the work needs.
template <class K>
int grid_bc(const GraphDev* g, K kernel, uint64_t items, uint64_t per_block) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kBcThreads, 0) != cudaSuccess || per_sm < 1)
    per_sm = 1;
  const uint64_t want = (items + per_block - 1) / per_block;
  return (int)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)g->sm_count * per_sm, want));
}

// One concurrent source lane: its stream and per-vertex state (parts of a
// BcSlab).
struct BcSlot {
  cudaStream_t s     = nullptr;
  BcVertex*    vx    = nullptr;
  double*      dsum  = nullptr;
  uint32_t*    order = nullptr;
  uint32_t*    vis   = nullptr;  // both copies
  BcLevel*     lv    = nullptr;  // device
  BcLevel*     hlv   = nullptr;  // pinned
  uint32_t     max_levels = 0;
  int          rc = NWG_OK;
  std::string  err;
};

// The memory of several lanes: one device and one pinned allocation (six of
// each lane's own took most of a first call).
struct BcSlab {
  unsigned char* dev  = nullptr;
  BcLevel*       host = nullptr;
};

constexpr uint64_t bc_align(uint64_t x) { return (x + 255) & ~uint64_t(255); }

// Offsets of a lane's arrays in its part of the slab; the last is its size.
struct BcLayout {
  uint64_t dsum, order, vis, lv, bytes;
  explicit BcLayout(uint64_t n) {
    dsum  = bc_align(n * sizeof(BcVertex));
    order = dsum + bc_align(n * 8);
    vis   = order + bc_align(n * 4);
    lv    = vis + bc_align(2 * ((n + 31) / 32) * 4);
    bytes = lv + bc_align((kBcBatch + 1) * sizeof(BcLevel));
  }
};

void slabs_free(std::vector<BcSlab>& slabs, std::vector<BcSlot>& slots) {
  for (auto& b : slots)
    if (b.s) {
      cudaStreamSynchronize(b.s);
      cudaStreamDestroy(b.s);
    }
  slots.clear();
  for (auto& x : slabs) {
    cudaFree(x.dev);
    if (x.host) cudaFreeHost(x.host);
  }
  slabs.clear();
}

// Adds `count` lanes to `slots`.  After a failure the caller frees them all.
int add_lanes(const GraphDev* g, std::vector<BcSlab>& slabs, std::vector<BcSlot>& slots, uint32_t count) {
  const uint64_t n = std::max<uint64_t>(g->n, 1);
  const BcLayout y(n);
  slabs.emplace_back();
  BcSlab& slab = slabs.back();
  if (cudaMalloc(&slab.dev, count * y.bytes) != cudaSuccess ||
      cudaMallocHost(&slab.host, count * (kBcBatch + 1) * sizeof(BcLevel)) != cudaSuccess) {
    cudaGetLastError();
    return set_error(NWG_ENOMEM, "betweenness workspace allocation failed");
  }
  for (uint32_t i = 0; i < count; ++i) {
    slots.emplace_back();
    BcSlot&        b = slots.back();
    unsigned char* d = slab.dev + i * y.bytes;
    b.vx             = reinterpret_cast<BcVertex*>(d);
    b.dsum           = reinterpret_cast<double*>(d + y.dsum);
    b.order          = reinterpret_cast<uint32_t*>(d + y.order);
    b.vis            = reinterpret_cast<uint32_t*>(d + y.vis);
    b.lv             = reinterpret_cast<BcLevel*>(d + y.lv);
    b.hlv            = slab.host + i * (kBcBatch + 1);
    NWG_CUDA_TRY(cudaStreamCreateWithFlags(&b.s, cudaStreamNonBlocking));
    NWG_CUDA_TRY(cudaMemsetAsync(b.dsum, 0, n * 8, b.s));
  }
  return NWG_OK;
}

}  // namespace

namespace nwg {

// The lanes, hub pieces and score array of a graph.  Making and freeing them
// took 14-25 ms of a call with 4 lanes on RMAT-20, so they are kept with the
// graph (up to 1 GB: 4 lanes of 2^23 vertices); a call beside another on the
// same graph makes its own.
struct BcWs {
  int                 device     = 0;
  uint64_t            kept_bytes = 0;
  std::vector<BcSlab> slabs;
  std::vector<BcSlot> slots;
  uint64_t*           piece[2]  = {nullptr, nullptr};  // out, in
  uint64_t            npiece[2] = {0, 0};
  bool                prepared  = false;  // pieces, use_in
  bool                use_in    = false;  // the in-CSR holds the out-CSR's edges, reversed
  float*              bc        = nullptr;  // scores, when the caller's array is on the host
  unsigned int*       maxbits   = nullptr;
  cudaEvent_t         ev0 = nullptr, ev1 = nullptr;
};

void bc_ws_free(BcWs* w) {
  if (!w) return;
  drop_bytes(w->device, w->kept_bytes);
  slabs_free(w->slabs, w->slots);
  for (auto* p : w->piece) cudaFree(p);
  cudaFree(w->bc);
  cudaFree(w->maxbits);
  if (w->ev0) cudaEventDestroy(w->ev0);
  if (w->ev1) cudaEventDestroy(w->ev1);
  delete w;
}

}  // namespace nwg

namespace {

// The hub pieces of one direction; synchronises.
int make_pieces(const GraphDev* g, const uint64_t* off, uint64_t m, uint64_t** piece, uint64_t* count) {
  const uint64_t cap = 2 * (m / kBcHub) + 1;  // a vertex of d > kBcHub edges has at most 2 d / kBcHub pieces
  if (cudaMalloc(piece, (cap + 1) * 8) != cudaSuccess) {
    cudaGetLastError();
    return set_error(NWG_ENOMEM, "betweenness hub list allocation failed");
  }
  auto* const c = reinterpret_cast<unsigned long long*>(*piece + cap);
  NWG_CUDA_TRY(cudaMemset(c, 0, 8));
  k_bc_pieces<<<grid_bc(g, k_bc_pieces, g->n, kBcThreads), kBcThreads>>>(off, g->n, *piece, cap, c);
  NWG_CUDA_TRY(cudaGetLastError());
  NWG_CUDA_TRY(cudaMemcpy(count, c, 8, cudaMemcpyDeviceToHost));
  *count = std::min<uint64_t>(*count, cap);
  return NWG_OK;
}

// The hub pieces and the comparison, on a graph's first call.
int prepare(GraphDev* g, BcWs& w) {
  int rc = make_pieces(g, g->off, g->m, &w.piece[0], &w.npiece[0]);
  if (!rc && g->in_off != g->off) rc = make_pieces(g, g->in_off, g->in_m, &w.piece[1], &w.npiece[1]);
  if (!rc) rc = csrs_transposed(g, nullptr, &w.use_in);
  if (rc) {
    for (auto*& p : w.piece) {
      cudaFree(p);
      p = nullptr;
    }
    return rc;
  }
  w.prepared = true;
  return NWG_OK;
}

// One source: forward levels in batches with one read-back each, then every
// backward level, then one synchronisation.
int run_source(const GraphDev* g, const BcWs& w, BcSlot& b, uint32_t s, float* bc) {
  const uint64_t n  = g->n;
  cudaStream_t   st = b.s;
  BcArgs         a;
  a.off       = g->off;
  a.col       = g->col;
  a.in_off    = g->in_off;
  a.in_col    = g->in_col;
  a.n         = n;
  a.m         = g->m;
  a.use_in    = w.use_in ? 1u : 0u;
  a.vx        = b.vx;
  a.dsum      = b.dsum;
  a.order     = b.order;
  a.vis[0]    = b.vis;
  a.vis[1]    = b.vis + (n + 31) / 32;
  a.lv        = b.lv;
  a.piece     = w.piece[0];
  a.npiece    = w.npiece[0];
  a.in_piece  = g->in_off == g->off ? w.piece[0] : w.piece[1];
  a.nin_piece = g->in_off == g->off ? w.npiece[0] : w.npiece[1];
  a.bc        = bc;
  k_bc_reset<<<grid_bc(g, k_bc_reset, std::max<uint64_t>(n, kBcThreads), kBcThreads), kBcThreads, 0, st>>>(a, s);
  NWG_CUDA_TRY(cudaGetLastError());
  std::vector<BcLevel> lv;  // every level
  const int gf = grid_bc(g, k_bc_forward, std::max(n, g->m / 32), kBcThreads);  // a step's grid: levels of any size
  for (uint32_t base = 0, done = 0, until = 8;;) {  // the first read-back after eight levels (hub graphs have 5-9)
    const uint32_t from = done;
    for (; done < until; ++done) k_bc_forward<<<gf, kBcThreads, 0, st>>>(a, done, base + done);
    NWG_CUDA_TRY(cudaGetLastError());
    NWG_CUDA_TRY(cudaMemcpyAsync(b.hlv, b.lv, (kBcBatch + 1) * sizeof(BcLevel), cudaMemcpyDeviceToHost, st));
    NWG_CUDA_TRY(cudaStreamSynchronize(st));
    for (uint32_t i = from; i < done && b.hlv[i].verts; ++i) lv.push_back(b.hlv[i]);
    if (b.hlv[done].verts == 0) break;
    if (done == kBcBatch) {
      k_bc_carry<<<1, 64, 0, st>>>(b.lv);
      base += kBcBatch;
      done = 0;
    }
    until = kBcBatch;
  }
  b.max_levels = std::max(b.max_levels, (uint32_t)lv.size());
  // eight lanes per vertex, and a warp per piece of the whole graph's list
  auto level_grid = [&](auto kernel, uint64_t verts, uint64_t pieces) {
    return grid_bc(g, kernel, std::max(verts, 4 * pieces), kBcThreads / 8);
  };
  for (size_t L = lv.size(); L-- > 0;) {
    const BcLevel& l = lv[L];
    bool           hubs_only = false;
    if (L + 1 < lv.size()) {
      const BcLevel& d = lv[L + 1];
      // a scattered edge costs a level gather and a double atomic, and its
      // dependencies a pass of their own
      if (a.use_in && 4 * d.in < l.out) {
        k_bc_scatter<<<level_grid(k_bc_scatter, d.verts, a.nin_piece), kBcThreads, 0, st>>>(a, d.first, d.verts,
                                                                                           (uint32_t)L);
      } else {
        k_bc_gather<<<level_grid(k_bc_gather, l.verts, a.npiece), kBcThreads, 0, st>>>(a, l.first, l.verts,
                                                                                       (uint32_t)L);
        if (a.npiece == 0) continue;
        hubs_only = true;
      }
    }
    k_bc_finish<<<grid_bc(g, k_bc_finish, l.verts, kBcThreads), kBcThreads, 0, st>>>(a, l.first, l.verts,
                                                                                     hubs_only ? 1u : 0u);
    NWG_CUDA_TRY(cudaGetLastError());
  }
  NWG_CUDA_TRY(cudaGetLastError());
  NWG_CUDA_TRY(cudaStreamSynchronize(st));
  return NWG_OK;
}

int bc_run(GraphDev* g, BcWs& w, const uint32_t* sources, uint32_t k, int normalize, uint32_t lanes,
           float* scores_host, float* scores_dev, nwg_bc_stats* stats) {
  const uint64_t n = g->n;
  if (!w.maxbits) NWG_CUDA_TRY(cudaMalloc(&w.maxbits, sizeof(unsigned int)));
  if (!w.ev0) NWG_CUDA_TRY(cudaEventCreate(&w.ev0));
  if (!w.ev1) NWG_CUDA_TRY(cudaEventCreate(&w.ev1));
  if (!w.prepared) {
    const int rc = prepare(g, w);
    if (rc) return rc;
  }
  float* bc = scores_dev;
  if (!bc) {
    if (!w.bc && cudaMalloc(&w.bc, std::max<uint64_t>(n, 1) * 4) != cudaSuccess) {
      cudaGetLastError();
      w.bc = nullptr;
      return set_error(NWG_ENOMEM, "betweenness score allocation failed");
    }
    bc = w.bc;
  }
  NWG_CUDA_TRY(cudaMemset(bc, 0, n * 4));
  NWG_CUDA_TRY(cudaMemset(w.maxbits, 0, sizeof(unsigned int)));
  int rc = NWG_OK;
  if (w.slots.size() < lanes) rc = add_lanes(g, w.slabs, w.slots, lanes - (uint32_t)w.slots.size());
  if (rc) return rc;
  for (uint32_t i = 0; i < lanes; ++i) {
    w.slots[i].rc         = NWG_OK;
    w.slots[i].max_levels = 0;
  }
  NWG_CUDA_TRY(cudaDeviceSynchronize());
  NWG_CUDA_TRY(cudaEventRecord(w.ev0, 0));
  std::atomic<uint32_t> next{0};
  auto                  lane_loop = [&, dev = g->device](BcSlot* bp) {
    cudaSetDevice(dev);
    for (uint32_t i = next++; i < k && bp->rc == NWG_OK; i = next++) {
      bp->rc = run_source(g, w, *bp, sources[i], bc);
      if (bp->rc) {
        char buf[512];
        nwg_last_error(buf, sizeof buf);
        bp->err = buf;
      }
    }
  };
  if (lanes == 1) {
    lane_loop(&w.slots[0]);  // one lane: the calling thread (profiler ranges stay on it)
  } else {
    std::vector<std::thread> th;
    for (uint32_t i = 0; i < lanes; ++i) th.emplace_back(lane_loop, &w.slots[i]);
    for (auto& t : th) t.join();
  }
  for (uint32_t i = 0; i < lanes; ++i)
    if (w.slots[i].rc && !rc) {
      rc = w.slots[i].rc;
      set_error(rc, w.slots[i].err);
    }
  if (!rc && normalize) {
    k_bc_max<<<grid_bc(g, k_bc_max, n, 256), 256>>>(bc, n, w.maxbits);
    k_bc_divide<<<grid_bc(g, k_bc_divide, n, 256), 256>>>(bc, n, w.maxbits);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) rc = cuda_error(e, "betweenness normalisation");
  }
  cudaEventRecord(w.ev1, 0);
  cudaError_t e = cudaDeviceSynchronize();
  if (!rc && e != cudaSuccess) rc = cuda_error(e, "betweenness");
  if (!rc && scores_host) {
    e = cudaMemcpy(scores_host, bc, n * 4, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) rc = cuda_error(e, "betweenness read-back");
  }
  if (stats) {
    nwg_bc_stats st = {};
    st.sources      = k;
    st.lanes        = lanes;
    for (uint32_t i = 0; i < lanes; ++i) st.max_levels = std::max(st.max_levels, w.slots[i].max_levels);
    cudaEventElapsedTime(&st.device_ms, w.ev0, w.ev1);
    *stats = st;
  }
  return rc;
}

}  // namespace

NWG_API int nwg_bc(nwg_graph h, const uint32_t* sources, uint32_t k, int normalize, uint32_t lanes, float* scores_host,
                   float* scores_dev, nwg_bc_stats* stats) {
  try {
    if (!h || (!sources && k)) return set_error(NWG_EINVAL, "NULL graph or sources");
    if (!scores_host && !scores_dev) return set_error(NWG_EINVAL, "no output array");
    auto* g = reinterpret_cast<GraphDev*>(h);
    for (uint32_t i = 0; i < k; ++i)
      if (sources[i] >= g->n) return set_error(NWG_EINVAL, "source " + std::to_string(sources[i]) + " >= n");
    if (lanes == 0) lanes = 4;
    lanes = std::min<uint32_t>(std::min<uint32_t>(lanes, 16), std::max<uint32_t>(k, 1));
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(g->device);
    struct Restore {
      int d;
      ~Restore() { cudaSetDevice(d); }
    } restore{prev};
    KeptState<BcWs, bc_ws_free> w(g->kept_mu, g->bc_ws);
    const int rc = bc_run(g, *w, sources, k, normalize, lanes, scores_host, scores_dev, stats);
    // (after an error a lane's dsum may not be zero)
    if (!rc)
      w.keep(g->device, w->slots.size() * BcLayout(g->n).bytes + (w->bc ? 4 * g->n : 0) +
                            8 * (2 * (g->m / kBcHub) + 2) * (w->piece[1] ? 2 : 1));
    return rc;
  } catch (const std::exception& ex) {
    return set_error(NWG_ENOMEM, std::string("betweenness failed: ") + ex.what());
  }
}
