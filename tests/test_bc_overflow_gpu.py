"""Betweenness where path counts pass the range of doubles: along a chain of k
diamonds the count doubles k times.  A last vertex whose count is infinite has
no successors, so its dependency is 0 and its predecessors' terms are count /
inf = 0: every score is finite, as in Brandes' computation in 64 bits
(test_bc_levels_gpu.py), within the 1e-6 on normalized scores used there.
Infinite counts further up give inf / inf: those scores, and the ones above
them, are NaN there and here."""
import numpy as np
import pytest

from oracle import graphgen as gg
from test_bc_levels_gpu import TOL, _bc64

pytestmark = pytest.mark.gpu


def _chain(k, mids, joined, clique=False):
    """k diamonds, then `mids` vertices behind the last, `joined` of which lead to one last vertex; the mids may form a clique."""
    a = 3 * np.arange(k, dtype=np.uint64)
    u = np.concatenate([a, a, a + 1, a + 2])
    v = np.concatenate([a + 1, a + 2, a + 3, a + 3])
    top = 3 * k
    mid = np.arange(top + 1, top + 1 + mids, dtype=np.uint64)
    last = top + 1 + mids
    u = np.concatenate([u, np.full(mids, top, np.uint64), mid[:joined]])
    v = np.concatenate([v, mid, np.full(joined, last, np.uint64)])
    if clique:
        x, y = np.triu_indices(mids, 1)
        u, v = np.concatenate([u, mid[x]]), np.concatenate([v, mid[y]])
    return gg.csr_from_pairs(u, v, last + 1)


CHAINS = {
    "gathered": lambda: _chain(1023, 2, 2),
    "scattered": lambda: _chain(1023, 12, 2, clique=True),  # the last level has far fewer in-edges than the one above out-edges
    "hub": lambda: _chain(1015, 600, 600),  # 600 * 2^1015 is past the range; its 600 edges are split into pieces
}


@pytest.mark.parametrize("name", sorted(CHAINS))
def test_last_vertex_with_an_infinite_count(nwg, name):
    off, cols = CHAINS[name]()
    g = nwg.Graph.from_csr(off, cols)
    with np.errstate(over="ignore"):
        want = _bc64(off, cols, [0])
    assert np.all(np.isfinite(want))
    got, _ = nwg.betweenness(g, np.array([0], np.uint32))
    assert np.max(np.abs(got - want)) <= TOL
    g.release()


def test_infinite_counts_above_the_last_level(nwg):
    off, cols = _chain(1050, 2, 2)
    g = nwg.Graph.from_csr(off, cols)
    raw, _ = nwg.betweenness(g, np.array([0], np.uint32), normalize=False)
    assert np.all(np.isnan(raw[: 3 * 1024]))  # from the source to the first infinite counts
    assert raw[-1] == 0
    g.release()
