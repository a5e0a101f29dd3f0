"""Marking steps of graphs without hubs, where the step that discovers most of
the graph offers parents to its targets instead of claiming them: vertex
counts that do not fill a word or a group of words, degrees that put the step
at different depths, directed pairs, parents arrays at any 4-byte boundary.
Depths, parents and the per-step trace equal the oracle's."""
import numpy as np
import pytest

from oracle import graphgen as gg

pytestmark = pytest.mark.gpu
NULL = 0xFFFFFFFF


@pytest.mark.parametrize("n", [32769, 40000, 65537, 100003, 262145])
@pytest.mark.parametrize("deg", [9, 14, 20, 32, 45])
def test_uniform_marking_steps(nwg, port, n, deg):
    import torch

    off, cols = gg.uniform(n, deg, seed=n + deg)
    in_off = in_cols = None
    if deg == 20:  # a directed pair: every other edge in one direction only
        keep = np.arange(cols.size) % 2 == 0
        src = np.repeat(np.arange(n, dtype=np.uint64), np.diff(off).astype(np.int64))
        off, cols = gg.directed_csr(src[keep], cols[keep].astype(np.uint64), n)
        in_off, in_cols = gg.transpose(off, cols, n)
    g = nwg.Graph.from_csr(off, cols, in_off, in_cols)
    for i, r in enumerate(map(int, gg.roots(off, 3, seed=deg))):
        parents, st = nwg.bfs(g, g, r, stats=True)
        want = port.depths(off, cols, r)
        assert np.array_equal(nwg.depths_from_parents(parents, r), want)
        assert np.array_equal(parents != NULL, want != NULL)
        assert port.verify(off, cols, r, parents, in_off, in_cols)
        _, tr = port.dobfs(off, cols, r, in_off, in_cols)
        got = st.trace()
        for key in ("dir", "found", "frontier"):
            assert np.array_equal(got[key], np.asarray(tr[key])[: got[key].size]), key
        buf = torch.full((n + 8,), 7, dtype=torch.int32, device="cuda")
        nwg.bfs_device(g, r, buf[i + 1:i + 1 + n])
        host = buf.cpu().numpy().view(np.uint32)
        assert port.verify(off, cols, r, host[i + 1:i + 1 + n], in_off, in_cols)
        assert np.all(host[: i + 1] == 7) and np.all(host[i + 1 + n:] == 7)
    g.release()
