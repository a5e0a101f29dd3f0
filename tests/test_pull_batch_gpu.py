"""Pulls on sparse graphs (average degree at most 4, where a pull probes
several candidates a lane at once) on the whole grid: tiles with few and many
candidates, lists of 3 to 6 and of 40 entries, vertex counts around the tile,
directed pairs.  Depths, parents and the per-step trace equal the oracle's."""
import numpy as np
import pytest

from oracle import graphgen as gg

pytestmark = pytest.mark.gpu
NULL = 0xFFFFFFFF


def _sparse(n, deg, hubs, seed, directed):
    rng = np.random.default_rng(seed)
    u, v = (rng.integers(0, n, n * deg // 2).astype(np.uint64) for _ in range(2))
    h = rng.integers(0, n, hubs).astype(np.uint64)  # a few vertices of about 40 more edges
    u, v = np.concatenate([u, np.repeat(h, 40)]), np.concatenate([v, rng.integers(0, n, 40 * hubs).astype(np.uint64)])
    if not directed:
        off, cols = gg.csr_from_pairs(u, v, n)
        return off, cols, None, None
    off, cols = gg.directed_csr(np.concatenate([u, v]), np.concatenate([v, u[::-1]]), n)
    return (off, cols, *gg.transpose(off, cols, n))


@pytest.mark.parametrize("n,deg,directed", [(40000, 4, False), (40001, 3, False), (65535, 4, True), (66049, 4, False), (131072, 2, False)])
def test_sparse_pulls(nwg, port, n, deg, directed):
    off, cols, in_off, in_cols = _sparse(n, deg, n // 2000, n, directed)
    g = nwg.Graph.from_csr(off, cols, in_off, in_cols)
    pulls = 0
    for r in map(int, gg.roots(off, 3, seed=deg)):
        for alpha, beta in ((15, 18), (100, 1000)):
            parents, st = nwg.bfs(g, g, r, 32, alpha, beta, stats=True)
            want = port.depths(off, cols, r)
            assert np.array_equal(nwg.depths_from_parents(parents, r), want)
            assert np.array_equal(parents != NULL, want != NULL)
            assert port.verify(off, cols, r, parents, in_off, in_cols)
            _, tr = port.dobfs(off, cols, r, in_off, in_cols, alpha=alpha, beta=beta)
            got = st.trace()
            for key in ("dir", "found", "frontier"):
                assert np.array_equal(got[key], np.asarray(tr[key])[: got[key].size]), key
            pulls += st.bu_steps
    assert pulls > 0
    g.release()
