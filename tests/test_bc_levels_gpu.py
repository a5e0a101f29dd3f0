"""Betweenness at the sizes where its work split changes: vertices of 512, 513
and many thousand edges (pieces), levels over several read-backs, levels that
pull and levels that scatter, a directed pair, and a directed graph registered
without an in-CSR (every level then pushes and gathers).  Within the 1e-6 on
normalized scores that the reference's BCVerifier states (see test_bc_gpu.py):
path counts are exact integers and a score's float sum over at most 5 sources
carries at most 5 * 2^-24 < 1e-6 relative.  The expected scores are Brandes'
in 64 bits: the C restatement sums a vertex's dependency in float, like the
reference, and is 2.6e-6 off them itself on a hub with 30,000 successors."""
import numpy as np
import pytest

from oracle import graphgen as gg

pytestmark = pytest.mark.gpu
TOL = 1e-6


def _bc64(off, cols, sources):
    n = off.size - 1
    src, dst = np.repeat(np.arange(n), np.diff(off).astype(np.int64)), cols.astype(np.int64)
    total = np.zeros(n)
    for root in sources:
        level, paths, steps = np.full(n, -1), np.zeros(n), []
        level[root], paths[root] = 0, 1.0
        while True:
            e = (level[src] == len(steps)) & (level[dst] == -1)
            if not e.any():
                break
            level[dst[e]] = len(steps) + 1
            np.add.at(paths, dst[e], paths[src[e]])
            steps.append((src[e], dst[e]))
        delta = np.zeros(n)
        for u, v in reversed(steps):
            np.add.at(delta, u, paths[u] / paths[v] * (1.0 + delta[v]))
        total += delta
    return total / total.max()


def _pair(n, m, seed):
    rng = np.random.default_rng(seed)
    u, v = (rng.integers(0, n, m).astype(np.uint64) for _ in range(2))
    return gg.directed_csr(u, v, n)


def _bowtie(k):
    """Two hubs of k leaves each, each joined to the same k // 2 middle vertices."""
    a, b = 0, 1
    mid = np.arange(2, 2 + k // 2, dtype=np.uint64)
    la = np.arange(mid[-1] + 1, mid[-1] + 1 + k, dtype=np.uint64)
    lb = la + np.uint64(k)
    u = np.concatenate([np.full(mid.size, a), np.full(mid.size, b), np.full(k, a), np.full(k, b)]).astype(np.uint64)
    return gg.csr_from_pairs(u, np.concatenate([mid, mid, la, lb]), int(lb[-1]) + 1)


GRAPHS = {
    "star512": lambda: gg.csr_from_pairs(np.zeros(512, np.uint64), np.arange(1, 513, dtype=np.uint64), 513),
    "star513": lambda: gg.csr_from_pairs(np.zeros(513, np.uint64), np.arange(1, 514, dtype=np.uint64), 514),
    "bowtie": lambda: _bowtie(20000),
    "path8": lambda: gg.csr_from_pairs(np.arange(7, dtype=np.uint64), np.arange(1, 8, dtype=np.uint64), 8),
    "path300": lambda: gg.csr_from_pairs(np.arange(299, dtype=np.uint64), np.arange(1, 300, dtype=np.uint64), 300),
    "grid": lambda: gg.grid(90, 75, 1, seed=1),
    "rmat15": lambda: gg.rmat(15, 16, seed=2),
    "uniform": lambda: gg.uniform(20011, 24, seed=3),
    "isolated": lambda: gg.csr_from_pairs(np.array([0], np.uint64), np.array([1], np.uint64), 70),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_bc_levels(nwg, name):
    off, cols = GRAPHS[name]()
    g = nwg.Graph.from_csr(off, cols)
    src = np.unique(np.concatenate([gg.roots(off, 3, seed=5), [0, g.n - 1]])).astype(np.uint32)
    want = _bc64(off, cols, src)
    for lanes in (1, 4, 1):  # kept lanes are reused
        got, _ = nwg.betweenness(g, src, lanes=lanes)
        assert np.max(np.abs(got - want)) <= TOL
    g.release()


@pytest.mark.parametrize("n,m", [(3000, 24000), (700, 300000)])
def test_bc_directed(nwg, n, m):
    off, cols = _pair(n, m, seed=n)
    in_off, in_cols = gg.transpose(off, cols, n)
    src = gg.roots(off, 5, seed=6)
    want = _bc64(off, cols, src)
    for extra in ((in_off, in_cols), ()):
        g = nwg.Graph.from_csr(off, cols, *extra)
        got, _ = nwg.betweenness(g, src)
        assert np.max(np.abs(got - want)) <= TOL
        g.release()
