// One whole direction-optimizing traversal by one block, its bitmaps in
// shared memory.  Included by nwg_dobfs.cu (inside namespace nwg).
//
// On a small graph a step moves a few kilobytes, and k_trav's steps cost a
// chain of L2 round trips plus a barrier of the whole grid: 4-28 us each on
// a B200, whatever their size.  One block needs __syncthreads() between
// steps, tests and claims bits in shared memory instead of L2, and makes the
// decision in every thread from shared counters; what is left of a step's
// chain is queue entry -> offsets -> columns.  Latency and one SM's loads in
// flight bound it, so it is used where the whole traversal is short (one
// graph: kBlkOneM) or where many traversals fill the SMs side by side (many
// roots of a graph, a ragged batch).
//
// The decisions are the reference's (nw::graph::bfs, bfs.hpp:186, 229, 241,
// 297-303) on the same counts as decide_on's, so directions, discoveries and
// frontier sizes per step are the same; a pull always runs as a pull.  The
// quotients of the switch rules are compared by multiplication: for
// integers, s > E / a exactly when s * a > E.
#pragma once

// Bitmaps of 2^19 vertices take 192 KB of the 227 KB a block may have.
constexpr uint64_t kBlkMaxN = 1ull << 19;
// Edge positions are 32-bit.
constexpr uint64_t kBlkMaxM = 1ull << 31;
// Vertices up to which the queue is in shared memory too.
constexpr uint32_t kBlkSmemQ = 2048;
constexpr int      kBlkTile  = 8;    // bitmap words per warp tile of a pull, at most (256 vertices)
constexpr int      kBlkBatch = 2;    // candidates a lane of a sparse graph's pull probes at once
constexpr int      kBlkVisit = 4;    // edges a lane tests per round of a push
constexpr uint32_t kBlkHub   = 512;  // a vertex of more out-edges is expanded by the whole block
constexpr uint32_t kBlkHubs  = 128;  // such vertices a step lists; further ones stay with their warp

struct BlkGraph {
  const uint64_t* off_;
  const uint32_t* col_;
  const uint64_t* in_off_;
  const uint32_t* in_col_;
  const uint32_t* Z;  // in-degree-zero bitmap, or NULL: such vertices' empty lists are looked at
  uint64_t        n;
  uint64_t        m;
  __device__ __forceinline__ uint32_t off(uint32_t v) const { return (uint32_t)__ldg(off_ + v); }
  __device__ __forceinline__ uint32_t col(uint32_t e) const { return __ldg(col_ + e); }
  __device__ __forceinline__ uint32_t in_off(uint32_t v) const { return (uint32_t)__ldg(in_off_ + v); }
  __device__ __forceinline__ uint32_t in_col(uint32_t e) const { return __ldg(in_col_ + e); }
};

// The same graph copied into shared memory.
struct BlkLocal {
  const uint32_t *off_, *col_, *in_off_, *in_col_;
  const uint32_t* Z;
  uint64_t        n;
  uint64_t        m;
  __device__ __forceinline__ uint32_t off(uint32_t v) const { return off_[v]; }
  __device__ __forceinline__ uint32_t col(uint32_t e) const { return col_[e]; }
  __device__ __forceinline__ uint32_t in_off(uint32_t v) const { return in_off_[v]; }
  __device__ __forceinline__ uint32_t in_col(uint32_t e) const { return in_col_[e]; }
};

// Queue entry, written by the step that discovers the vertex: its offsets
// are loaded once, there, and the next push starts from one 16-byte load.
// A vertex is queued at most once per traversal, so one array of n entries
// serves all levels: a level's frontier is a range of it, its discoveries
// are appended behind.
struct alignas(16) BlkEnt {
  uint32_t v, deg, lo, pad;  // out-edges [lo, lo + deg)
};

// Shared memory of one traversal, in front of its bitmaps (and queue).
template <int T>
struct BlkSmem {
  uint32_t cnt;    // discoveries of the step
  uint32_t scout;  // their out-degree sum
  uint32_t nhub;
  uint32_t hub[kBlkHubs];  // queue indices of the step's hubs
  union {
    struct {  // a push's group of up to 32 queue entries
      uint32_t pre[32];   // exclusive prefix of the out-degrees
      uint32_t base[32];  // lo minus prefix: edge e of the group is column base + e
      uint32_t u[32];
    } grp[T / 32];
    uint16_t cand[T / 32][kBlkTile * 32];  // a pull tile's candidates (local vertex indices)
  };
};

__host__ __device__ inline uint64_t blk_bitmap_bytes(uint64_t n) { return 3 * (((n + 31) / 32 + 3) & ~3ull) * 4; }

template <int T>
__host__ __device__ constexpr size_t blk_fixed_bytes() {
  return (sizeof(BlkSmem<T>) + 15) & ~size_t(15);
}

template <int T>
inline size_t blk_smem_bytes(uint64_t n) {
  return blk_fixed_bytes<T>() + blk_bitmap_bytes(n) + (n <= kBlkSmemQ ? n * sizeof(BlkEnt) : 0);
}

// A graph of at most this many bytes beside its traversal's state is copied
// into shared memory first (bytes of the copy: blk_local_bytes).
constexpr size_t kBlkLocalMax = 220 * 1024;
inline size_t blk_local_bytes(uint64_t n, uint64_t m, bool symmetric) {
  const size_t one = ((n + 1 + 3) & ~3ull) * 4 + ((m + 3) & ~3ull) * 4;
  return symmetric ? one : 2 * one;
}

// Copies g to `at` (16-byte aligned, blk_local_bytes); ends with a barrier.
// One SM reads RMAT-10 (94 KB) in about a microsecond; a step's loads then
// take a shared-memory access instead of an L2 one.
template <int T>
__device__ __forceinline__ BlkLocal blk_copy(const BlkGraph& g, unsigned char* at) {
  const uint32_t n = (uint32_t)g.n, m = (uint32_t)g.m;
  const bool     one = g.in_off_ == g.off_ && g.in_col_ == g.col_;
  uint32_t*      d   = reinterpret_cast<uint32_t*>(at);
  BlkLocal       l{d, nullptr, nullptr, nullptr, g.Z, g.n, g.m};
  auto           csr = [&](const uint64_t* off, const uint32_t* col, uint32_t* to) -> uint32_t* {
    uint32_t* const tc = to + ((n + 1 + 3) & ~3u);
    for (uint32_t i = threadIdx.x; i <= n; i += T) to[i] = (uint32_t)__ldg(off + i);
    if ((reinterpret_cast<uintptr_t>(col) & 15) == 0) {
      for (uint32_t i = threadIdx.x; i < m / 4; i += T)
        reinterpret_cast<uint4*>(tc)[i] = __ldg(reinterpret_cast<const uint4*>(col) + i);
      for (uint32_t i = (m & ~3u) + threadIdx.x; i < m; i += T) tc[i] = __ldg(col + i);
    } else {
      for (uint32_t i = threadIdx.x; i < m; i += T) tc[i] = __ldg(col + i);
    }
    return tc;
  };
  uint32_t* const c = csr(g.off_, g.col_, d);
  l.col_            = c;
  l.in_off_         = d;
  l.in_col_         = c;
  if (!one) {
    uint32_t* const e = c + ((m + 3) & ~3u);
    l.in_off_         = e;
    l.in_col_         = csr(g.in_off_, g.in_col_, e);
  }
  __syncthreads();
  return l;
}

// Enough for every graph of at most nmax vertices (a graph with its queue in
// shared memory may need more than a larger one).
template <int T>
inline size_t blk_smem_bytes_upto(uint64_t nmax) {
  return std::max(blk_smem_bytes<T>(nmax), blk_smem_bytes<T>(std::min<uint64_t>(nmax, kBlkSmemQ)));
}

// One round of edge tests (bfs.hpp:280-289): the lane's edges u[k] -> v[k],
// kNull = none.  A claim's winner writes the parent and appends the vertex
// with its offsets, one counter update per warp.  All lanes call.
template <int T, class G>
__device__ __forceinline__ void blk_visit(BlkSmem<T>& sm, const G& g, const uint32_t (&u)[kBlkVisit],
                                          const uint32_t (&v)[kBlkVisit], uint32_t* V, uint32_t* parents,
                                          BlkEnt* out, uint32_t& scout) {
  const unsigned lane = threadIdx.x & 31;
  uint32_t       win  = 0;
#pragma unroll
  for (int k = 0; k < kBlkVisit; ++k) {
    if (v[k] == kNull) continue;
    const uint32_t bit = 1u << (v[k] & 31);
    if (!(V[v[k] >> 5] & bit) && !(atomicOr(V + (v[k] >> 5), bit) & bit)) win |= 1u << k;
  }
  if (!__any_sync(kFullMask, win)) return;
  uint32_t lo[kBlkVisit], hi[kBlkVisit];
#pragma unroll
  for (int k = 0; k < kBlkVisit; ++k) {
    lo[k] = hi[k] = 0;
    if (win & (1u << k)) {
      lo[k] = g.off(v[k]);
      hi[k] = g.off(v[k] + 1);
    }
  }
  const uint32_t mine = __popc(win);
  const uint32_t inc  = warp_incl_scan(mine);
  uint32_t       slot = 0;
  if (lane == 31) slot = atomicAdd(&sm.cnt, inc);
  slot = __shfl_sync(kFullMask, slot, 31) + inc - mine;
#pragma unroll
  for (int k = 0; k < kBlkVisit; ++k)
    if (win & (1u << k)) {
      parents[v[k]] = u[k];
      out[slot++]   = BlkEnt{v[k], hi[k] - lo[k], lo[k], 0u};
      scout += hi[k] - lo[k];
    }
}

// One top-down step over queue entries [b, e) (bfs.hpp:242-295), discoveries
// to out[0 ...).  Warps take groups of up to 32 entries (fewer when the
// frontier is small, so that every warp has one) and deal the group's edges
// to their lanes by a prefix of the degrees; no barrier between groups, so
// warps hide each other's latency.  Vertices of more than kBlkHub out-edges
// are listed and then expanded by all threads.  Adds to sm.cnt, sm.scout.
template <int T, class G>
__device__ __forceinline__ void blk_push(BlkSmem<T>& sm, const G& g, const BlkEnt* q, uint32_t b, uint32_t e,
                                         BlkEnt* out, uint32_t* V, uint32_t* parents) {
  const unsigned lane  = threadIdx.x & 31, wib = threadIdx.x >> 5;
  auto&          grp   = sm.grp[wib];
  uint32_t       scout = 0;
  const uint32_t gs    = min(32u, (e - b + T / 32 - 1) / (T / 32));
  for (uint32_t g0 = b + wib * gs; g0 < e; g0 += (T / 32) * gs) {
    BlkEnt x{0, 0, 0, 0};
    if (lane < gs && g0 + lane < e) {
      x = q[g0 + lane];
      if (x.deg > kBlkHub) {
        const uint32_t h = atomicAdd(&sm.nhub, 1u);
        if (h < kBlkHubs) {
          sm.hub[h] = g0 + lane;
          x.deg     = 0;
        }
      }
    }
    const uint32_t inc = warp_incl_scan(x.deg);
    const uint32_t tot = __shfl_sync(kFullMask, inc, 31);
    grp.pre[lane]      = inc - x.deg;
    grp.base[lane]     = x.lo - (inc - x.deg);
    grp.u[lane]        = x.v;
    __syncwarp();
    for (uint32_t e0 = 0; e0 < tot; e0 += 32 * kBlkVisit) {
      uint32_t u[kBlkVisit], v[kBlkVisit];
#pragma unroll
      for (int k = 0; k < kBlkVisit; ++k) {
        const uint32_t i = e0 + k * 32 + lane;
        u[k]             = 0;
        v[k]             = kNull;
        if (i < tot) {  // owner: the last entry whose prefix is at most i
          int o = 0;
#pragma unroll
          for (int s = 16; s >= 1; s >>= 1)
            if (grp.pre[o + s] <= i) o += s;
          u[k] = grp.u[o];
          v[k] = g.col(grp.base[o] + i);
        }
      }
      blk_visit<T>(sm, g, u, v, V, parents, out, scout);
    }
    __syncwarp();
  }
  __syncthreads();
  const uint32_t nh = min(sm.nhub, kBlkHubs);
  for (uint32_t h = 0; h < nh; ++h) {
    const BlkEnt x = q[sm.hub[h]];
    for (uint32_t e0 = threadIdx.x & ~31u; e0 < x.deg; e0 += T * kBlkVisit) {
      uint32_t u[kBlkVisit], v[kBlkVisit];
#pragma unroll
      for (int k = 0; k < kBlkVisit; ++k) {
        const uint32_t i = e0 + k * T + lane;
        u[k]             = x.v;
        v[k]             = i < x.deg ? g.col(x.lo + i) : kNull;
      }
      blk_visit<T>(sm, g, u, v, V, parents, out, scout);
    }
  }
  scout = __reduce_add_sync(kFullMask, scout);
  if (lane == 0 && scout) atomicAdd(&sm.scout, scout);
}

// One pull (bfs.hpp:211-228) over `front` into the discovery bitmap N, as
// bu_step: a warp takes tiles of tw bitmap words, compacts their unvisited
// vertices and streams them through its lanes; each lane has the next
// candidate's offsets loading and tests kBuProbe in-edges per round.  On
// sparse graphs, most of whose lists one probe covers (kSparse), kBlkBatch
// candidates a lane are probed straight through first and only longer lists
// without a hit are streamed (a 512 x 512 grid 1.70 -> 1.63 ms, 1,024 mixed
// items 2.11 -> 1.99 ms).  Lists longer than kBuLane go to the warp.  V is only
// read.  Adds the discoveries to sm.cnt.
template <int T, bool kSparse, class G>
__device__ __forceinline__ void blk_pull(BlkSmem<T>& sm, const G& g, const uint32_t* V, const uint32_t* front,
                                         uint32_t* N, uint32_t* parents, uint32_t nwords) {
  const unsigned  lane    = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const unsigned  lt_mask = (1u << lane) - 1u;
  uint16_t* const cand    = sm.cand[wib];
  // small graphs: fewer words per tile, so that every warp has one
  const uint32_t tw    = min((uint32_t)kBlkTile, (nwords + T / 32 - 1) / (T / 32));
  const uint32_t tail   = (uint32_t)(g.n & 31);
  constexpr uint32_t probed = kSparse ? kBuProbe : 0;
  uint32_t       awake  = 0;
  for (uint32_t w0 = wib * tw; w0 < nwords; w0 += (T / 32) * tw) {
    const uint32_t w  = w0 + lane;
    const bool     wv = lane < tw && w < nwords;
    uint32_t       cm = 0;
    if (wv) {
      cm = ~V[w];
      if (g.Z) cm &= ~__ldg(g.Z + w);
      if (w == nwords - 1 && tail) cm &= (1u << tail) - 1u;
      N[w] = 0;
    }
    uint32_t       total = compact_tile(cm, cand);
    const uint32_t vbase = w0 * 32;
    uint32_t       rest  = kSparse ? 0u : total;  // candidates left for the streaming scan
    for (uint32_t j = 0; kSparse && j < total; j += 32 * kBlkBatch) {
      uint32_t c[kBlkBatch], b[kBlkBatch], d[kBlkBatch], x[kBlkBatch][kBuProbe];
#pragma unroll
      for (int q = 0; q < kBlkBatch; ++q) {
        const uint32_t i = j + q * 32 + lane;
        c[q]             = vbase + (i < total ? cand[i] : 0u);
        b[q]             = g.in_off(c[q]);
        d[q]             = i < total ? g.in_off(c[q] + 1) - b[q] : 0u;
      }
#pragma unroll
      for (int q = 0; q < kBlkBatch; ++q)
#pragma unroll
        for (int k = 0; k < kBuProbe; ++k) x[q][k] = k < d[q] ? g.in_col(b[q] + k) : kNull;
      __syncwarp();  // this batch's candidates are read; the list is refilled from its start
#pragma unroll
      for (int q = 0; q < kBlkBatch; ++q) {
        uint32_t par = kNull;
#pragma unroll
        for (int k = kBuProbe - 1; k >= 0; --k)  // the first hit in row order stays
          if (x[q][k] != kNull && ((front[x[q][k] >> 5] >> (x[q][k] & 31)) & 1u)) par = x[q][k];
        if (par != kNull) {
          parents[c[q]] = par;
          atomicOr(N + (c[q] >> 5), 1u << (c[q] & 31));
        }
        const bool     more = par == kNull && d[q] > kBuProbe;
        const unsigned m    = __ballot_sync(kFullMask, more);
        if (more) cand[rest + __popc(m & lt_mask)] = (uint16_t)(c[q] - vbase);
        rest += __popc(m);
      }
    }
    if (kSparse) __syncwarp();
    total = rest;
    // current candidate (cu, next in-edge ce, end cend, first in-edge cb)
    // and the next one (nu; offsets in flight)
    uint32_t cu = 0, ce = 0, cend = 0, cb = 0, nu = 0, nb = 0, nend = 0;
    bool     cv = lane < total, nv = false;
    if (cv) {
      cu   = vbase + cand[lane];
      cb   = g.in_off(cu);
      ce   = cb + probed;
      cend    = g.in_off(cu + 1);
    }
    uint32_t ptr = min(total, 32u);  // next unassigned list entry (warp-uniform)
    if (ptr + lane < total) {
      nu   = vbase + cand[ptr + lane];
      nb   = g.in_off(nu);
      nend = g.in_off(nu + 1);
      nv   = true;
    }
    ptr = min(total, ptr + 32u);
    while (__any_sync(kFullMask, cv)) {
      bool     found = false, handoff = false;
      uint32_t par   = 0;
      if (cv) {
        uint32_t nbv[kBuProbe];
#pragma unroll
        for (int k = 0; k < kBuProbe; ++k) nbv[k] = ce + k < cend ? g.in_col(ce + k) : kNull;
#pragma unroll
        for (int k = kBuProbe - 1; k >= 0; --k)  // the first hit in row order stays
          if (nbv[k] != kNull && ((front[nbv[k] >> 5] >> (nbv[k] & 31)) & 1u)) {
            par   = nbv[k];
            found = true;
          }
        if (!found) {
          ce += kBuProbe;
          if (ce >= cend) cv = false;
          else if (ce - cb >= kBuLane) handoff = true;
        }
      }
      unsigned pend = __ballot_sync(kFullMask, handoff);
      while (pend) {
        const int leader = __ffs(pend) - 1;
        pend &= pend - 1;
        const uint32_t b  = __shfl_sync(kFullMask, ce, leader);
        const uint32_t en = __shfl_sync(kFullMask, cend, leader);
        bool           lf = false;
        uint32_t       lp = 0;
        for (uint32_t base = b; base < en; base += 32) {
          const uint32_t i = base + lane;
          uint32_t       x = 0;
          bool           h = false;
          if (i < en) {
            x = g.in_col(i);
            h = (front[x >> 5] >> (x & 31)) & 1u;
          }
          const unsigned hm = __ballot_sync(kFullMask, h);
          if (hm) {
            lp = __shfl_sync(kFullMask, x, __ffs(hm) - 1);
            lf = true;
            break;
          }
        }
        if ((int)lane == leader) {
          found = lf;
          par   = lp;
          cv    = false;
        }
      }
      if (found) {
        parents[cu] = par;
        atomicOr(N + (cu >> 5), 1u << (cu & 31));
        cv = false;
      }
      if (!cv && nv) {
        cu   = nu;
        cb   = nb;
        ce   = nb + probed;
        cend    = nend;
        cv   = true;
        nv   = false;
      }
      if (ptr < total) {  // warp-uniform
        const unsigned need = __ballot_sync(kFullMask, !nv);
        const uint32_t at   = ptr + __popc(need & lt_mask);
        if (!nv && at < total) {
          nu   = vbase + cand[at];
          nb   = g.in_off(nu);
          nend = g.in_off(nu + 1);
          nv   = true;
        }
        ptr = min(total, ptr + (uint32_t)__popc(need));
      }
    }
    __syncwarp();
    if (wv) awake += __popc(N[w]);
    __syncwarp();
  }
  awake = __reduce_add_sync(kFullMask, awake);
  if (lane == 0 && awake) atomicAdd(&sm.cnt, awake);
}

// The set bits of F as queue entries (bfs.hpp:235-239).
template <int T, class G>
__device__ __forceinline__ void blk_b2q(BlkSmem<T>& sm, const G& g, const uint32_t* F, uint32_t nwords,
                                        BlkEnt* out) {
  const unsigned lane = threadIdx.x & 31;
  for (uint32_t w0 = threadIdx.x & ~31u; w0 < nwords; w0 += T) {
    const uint32_t w    = w0 + lane;
    uint32_t       x    = w < nwords ? F[w] : 0u;
    const uint32_t inc  = warp_incl_scan((uint32_t)__popc(x));
    uint32_t       slot = 0;
    if (lane == 31 && inc) slot = atomicAdd(&sm.cnt, inc);
    slot = __shfl_sync(kFullMask, slot, 31) + inc - __popc(x);
    while (x) {
      const uint32_t v  = w * 32 + (__ffs(x) - 1);
      const uint32_t lo = g.off(v);
      out[slot++]       = BlkEnt{v, g.off(v + 1) - lo, lo, 0u};
      x &= x - 1;
    }
  }
}

// The whole traversal from `root` by the calling block of T threads.  smem:
// blk_smem_bytes<T>(n) bytes, 16-byte aligned.  q: n entries, not used where
// n <= kBlkSmemQ.  trace: control block whose per-step trace is written, or
// NULL.  All threads return the result; a barrier must come before the
// block's next traversal.
template <int T, class G>
__device__ __forceinline__ RaggedResult block_traverse(const G& g, uint32_t root, uint32_t alpha, uint32_t beta,
                                                       bool topdown_only, uint32_t* parents, BlkEnt* q,
                                                       unsigned char* smem, Ctrl* trace, uint32_t* trace_len) {
  BlkSmem<T>&    sm     = *reinterpret_cast<BlkSmem<T>*>(smem);
  const uint32_t n      = (uint32_t)g.n;
  const uint32_t nwords = (n + 31) / 32;
  const uint32_t wpad   = (nwords + 3) & ~3u;
  uint32_t*      V      = reinterpret_cast<uint32_t*>(smem + blk_fixed_bytes<T>());
  uint32_t*      F      = V + wpad;
  uint32_t*      N      = F + wpad;
  BlkEnt* const  ent    = n <= kBlkSmemQ ? reinterpret_cast<BlkEnt*>(N + wpad) : q;
  const bool     t0     = threadIdx.x == 0;
  const unsigned long long t_start = trace ? globaltimer() : 0ull;
  uint32_t                 ntr     = 0;
  auto tr = [&](uint8_t dir, uint64_t frontier, uint64_t found) {
    if (trace && ntr < NWG_TRACE_CAP) {
      if (t0) {
        trace->trace_dir[ntr]      = dir;
        trace->trace_frontier[ntr] = frontier;
        trace->trace_found[ntr]    = found;
        trace->trace_end_ns[ntr]   = globaltimer() - t_start;
      }
      ++ntr;
    }
  };
  auto restart = [&]() {  // the step's counters; between barriers
    if (t0) sm.cnt = sm.scout = sm.nhub = 0;
  };

  const uint32_t rlo = g.off(root), rdeg = g.off(root + 1) - rlo;
  for (uint32_t w = threadIdx.x; w < nwords; w += T) V[w] = w == (root >> 5) ? 1u << (root & 31) : 0u;
  // parents := null except the root (bfs.hpp:175, 180), 16 bytes at a time
  // between the row's unaligned ends
  {
    const uint32_t head = min(n, (uint32_t)((4 - ((reinterpret_cast<uintptr_t>(parents) >> 2) & 3)) & 3));
    const uint32_t n4   = (n - head) >> 2;
    uint4* const   p4   = reinterpret_cast<uint4*>(parents + head);
    for (uint32_t i = threadIdx.x; i < n4; i += T) p4[i] = make_uint4(kNull, kNull, kNull, kNull);
    if (threadIdx.x < head) parents[threadIdx.x] = kNull;
    for (uint32_t i = head + 4 * n4 + threadIdx.x; i < n; i += T) parents[i] = kNull;
  }
  restart();
  if (t0) ent[0] = BlkEnt{root, rdeg, rlo, 0u};
  __syncthreads();
  if (t0) parents[root] = root;
  if (t0 && trace) trace->t_first_decide = globaltimer() - t_start;

  RaggedResult r      = {};
  uint64_t     echeck = g.m;   // edges_to_check, bfs.hpp:177
  uint64_t     scout  = rdeg;  // bfs.hpp:178
  uint32_t     qb = 0, qe = 1;  // the frontier: ent[qb, qe)
  r.levels            = 1;
  r.reached           = 1;
  for (;;) {
    if (!topdown_only && scout * alpha > echeck) {  // bfs.hpp:186
      uint32_t awake = qe - qb, old;
      bool     first = true;
      do {
        old = awake;
        if (g.m < (kBuProbe + 1) * g.n) blk_pull<T, true>(sm, g, V, first ? V : F, N, parents, nwords);
        else blk_pull<T, false>(sm, g, V, first ? V : F, N, parents, nwords);
        __syncthreads();
        awake = sm.cnt;
        for (uint32_t w = threadIdx.x; w < nwords; w += T) V[w] |= N[w];
        __syncthreads();
        restart();
        tr(1, old, awake);
        r.bu_steps++;
        r.reached += awake;
        if (awake) r.levels++;
        uint32_t* const x = F;
        F                 = N;  // the latest pull's discoveries
        N                 = x;
        first             = false;
        __syncthreads();
      } while (awake >= old || (uint64_t)awake * beta > n);  // bfs.hpp:229
      if (!awake) break;                                     // bfs.hpp:231-233
      blk_b2q<T>(sm, g, F, nwords, ent + qe);
      qb    = qe;
      qe    = qb + awake;
      scout = 1;  // bfs.hpp:241
      r.b2q_steps++;
      __syncthreads();
      restart();
      __syncthreads();
      continue;
    }
    echeck -= scout;  // bfs.hpp:243
    blk_push<T>(sm, g, ent, qb, qe, ent + qe, V, parents);
    __syncthreads();
    const uint32_t found = sm.cnt;
    scout                = sm.scout;  // bfs.hpp:271
    tr(0, qe - qb, found);
    r.td_steps++;
    r.reached += found;
    if (!found) break;  // all next bins empty, bfs.hpp:297-303
    r.levels++;
    qb = qe;
    qe = qb + found;
    __syncthreads();
    restart();
    __syncthreads();
  }
  r.steps = r.td_steps + r.bu_steps + r.b2q_steps;
  if (trace_len) *trace_len = ntr;
  return r;
}
