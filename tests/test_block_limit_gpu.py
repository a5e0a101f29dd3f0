"""Graphs around the line between one block and the whole grid for a single
traversal (at most 24,576 vertices with edges or 6.5 entries for each, at
most 2^15 vertices and 2^18 entries), so that both run next to it: depths,
parents and per-step traces equal the oracle's, for parents in host memory, in
device memory and without an allocation."""
import numpy as np
import pytest

from oracle import graphgen as gg

pytestmark = pytest.mark.gpu
NULL = 0xFFFFFFFF


def _ring(n, active, degree):
    """`active` of n vertices on a ring, each joined to those degree / 2 distances away."""
    v = np.repeat(np.arange(active, dtype=np.uint64), degree // 2)
    step = 1 + np.random.default_rng(active).choice(active // 2 - 1, degree // 2, replace=False).astype(np.uint64)
    return gg.csr_from_pairs(v, (v + np.tile(step, active)) % active, n)


GRAPHS = [(24576, 24576, 8), (24577, 24577, 8), (1 << 15, 24576, 8), (1 << 15, 24577, 8), (1 << 15, 1 << 15, 6),
          ((1 << 15) + 1, (1 << 15) + 1, 4), (20000, 20000, 12), (21846, 21846, 12)]


@pytest.mark.parametrize("n,active,degree", GRAPHS)
def test_around_the_limit(nwg, port, n, active, degree):
    import torch

    off, cols = _ring(n, active, degree)
    assert cols.size == active * degree
    g = nwg.Graph.from_csr(off, cols)
    dev = torch.empty(n, dtype=torch.int32, device="cuda")
    arrays = [torch.from_numpy(off.view(np.int64)).cuda(), torch.from_numpy(cols.view(np.int32)).cuda()]
    for r in (0, active - 1, n - 1):
        want = port.depths(off, cols, r)
        _, tr = port.dobfs(off, cols, r)
        parents, st = nwg.bfs(g, root=r, stats=True)
        nwg.bfs_device(g, r, dev)
        on_device = dev.cpu().numpy().view(np.uint32)
        nwg.bfs_noalloc(*arrays, n, r, dev)
        for p in (parents, on_device, dev.cpu().numpy().view(np.uint32)):
            assert np.array_equal(p != NULL, want != NULL)
            assert port.verify(off, cols, r, p)
        got = st.trace()
        m = got["dir"].size
        assert m == min(len(tr["dir"]), 256) and st.status == 0
        for key in ("dir", "found", "frontier"):
            assert np.array_equal(got[key], np.asarray(tr[key])[:m]), key
    g.release()
