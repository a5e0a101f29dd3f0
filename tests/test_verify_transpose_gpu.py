"""The device verifier on graphs whose in-CSR is not the transpose of their
out-CSR: directed graphs registered without an in-CSR, and pairs with a wrong
one.  Depths come from the out-graph alone (bfs.hpp:47-63), so the verdict,
the vertex, the reason, the reached vertices and the levels equal the
reference's (restated in test_verify_gpu.py), also for the parents that a
traversal over the same in-CSR returns."""
import numpy as np
import pytest

from oracle import graphgen as gg
from test_verify_gpu import reference_verdict

pytestmark = pytest.mark.gpu
NULL = 0xFFFFFFFF


def _star(n):
    """Arcs from 0 to every other vertex, none back."""
    return gg.directed_csr(np.zeros(n - 1, np.uint64), np.arange(1, n, dtype=np.uint64), n)


def _one_way(n):
    """Root 0 and vertices joined both ways, and a last vertex with an arc to the root only."""
    rng = np.random.default_rng(n)
    u, v = (rng.integers(0, n - 1, 4 * n).astype(np.uint64) for _ in range(2))
    first = np.arange(1, n - 1, dtype=np.uint64)
    zero = np.zeros(n - 2, np.uint64)
    return gg.directed_csr(np.concatenate([u, v, zero, first, [n - 1]]).astype(np.uint64),
                           np.concatenate([v, u, first, zero, [0]]).astype(np.uint64), n)


def _random(n, m):
    rng = np.random.default_rng(m)
    return gg.directed_csr(*(rng.integers(0, n, m).astype(np.uint64) for _ in range(2)), n)


def _hubs(k, leaves):
    """A root with arcs to k hubs, each with arcs to the same leaves."""
    hub = np.arange(1, k + 1, dtype=np.uint64)
    leaf = np.arange(k + 1, k + 1 + leaves, dtype=np.uint64)
    u = np.concatenate([np.zeros(k, np.uint64), np.repeat(hub, leaves)])
    return gg.directed_csr(u, np.concatenate([hub, np.tile(leaf, k)]), k + 1 + leaves)


GRAPHS = {
    "star1024": lambda: _star(1024),
    "star40000": lambda: _star(40000),
    "one_way": lambda: _one_way(3000),
    "random": lambda: _random(4000, 60000),
    "hubs": lambda: _hubs(70, 3000),
}


def _same(nwg, port, g, off, cols, root, parents, in_off, in_cols):
    want = reference_verdict(port, off, cols, root, parents, in_off, in_cols)
    got = nwg.verify(g, root, parents)
    assert bool(got.valid) == want[0]
    if not want[0]:
        assert (got.first_bad, got.reason) == (want[1], want[2])
    depth = port.depths(off, cols, root)
    assert got.reached == np.count_nonzero(depth != NULL)
    assert got.levels == depth[depth != NULL].max() + 1


@pytest.mark.parametrize("pair", ["none", "wrong", "wrong_device", "transpose"])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_verdicts_do_not_rest_on_the_in_csr(nwg, port, name, pair):
    off, cols = GRAPHS[name]()
    n = off.size - 1
    in_off = in_cols = None
    if pair != "none":
        in_off, in_cols = gg.transpose(off, cols, n)
    if pair.startswith("wrong"):  # the transpose with every vertex renamed to the next
        src = np.repeat(np.arange(n, dtype=np.uint64), np.diff(in_off).astype(np.int64))
        in_off, in_cols = gg.directed_csr((src + 1) % n, (in_cols.astype(np.uint64) + 1) % n, n)
    keep = None
    if pair == "wrong_device":
        import torch

        keep = [torch.from_numpy(np.ascontiguousarray(x).view(np.int64 if x.itemsize == 8 else np.int32)).cuda()
                for x in (off, cols, in_off, in_cols)]
        g = nwg.Graph.from_csr(*keep, device=True)
    else:
        g = nwg.Graph.from_csr(off, cols, in_off, in_cols)
    for root in (0, int(gg.roots(off, 1, seed=2)[0])):
        true, _ = port.dobfs(off, cols, root, *gg.transpose(off, cols, n))
        mine = nwg.bfs(g, root=root)  # rests on the pair it was given
        for parents in (true, mine):
            _same(nwg, port, g, off, cols, root, parents, in_off, in_cols)
    g.release()
