"""The device verifier's own traversal and long in-lists: levels over several
read-backs, pushes after pulls, a hub whose parent is the last of thousands of
in-neighbours (its list is checked in pieces by the grid), and planted
mistakes there.  Verdicts equal the reference's (restated in
test_verify_gpu.py)."""
import numpy as np
import pytest

from oracle import graphgen as gg
from test_verify_gpu import reference_verdict

pytestmark = pytest.mark.gpu
NULL = 0xFFFFFFFF


def _same(nwg, port, g, off, cols, root, parents):
    want = reference_verdict(port, off, cols, root, parents)
    got = nwg.verify(g, root, parents)
    assert bool(got.valid) == want[0]
    if not want[0]:
        assert (got.first_bad, got.reason) == (want[1], want[2])
    depth = port.depths(off, cols, root)
    assert got.reached == np.count_nonzero(depth != NULL)
    assert got.levels == depth[depth != NULL].max() + 1


@pytest.mark.parametrize("leaves", [31, 33, 1055, 1056, 1057, 2081, 30000])
def test_hub_whose_parent_is_last_in_its_list(nwg, port, leaves):
    # hub 0 joined to leaves 1..leaves and to the root, whose id is the largest but two; an isolated pair behind
    root = leaves + 1
    u = np.concatenate([np.zeros(leaves + 1, np.uint64), [root + 1]]).astype(np.uint64)
    v = np.concatenate([np.arange(1, leaves + 2), [root + 2]]).astype(np.uint64)
    off, cols = gg.csr_from_pairs(u, v, root + 3)
    g = nwg.Graph.from_csr(off, cols)
    parents, _ = port.dobfs(off, cols, root)
    assert parents[0] == root
    _same(nwg, port, g, off, cols, root, parents)
    for wrong in (1, root + 1):  # an in-neighbour one level down; not an in-neighbour
        bad = parents.copy()
        bad[0] = wrong
        _same(nwg, port, g, off, cols, root, bad)
    _same(nwg, port, g, off, cols, root, parents)  # nothing is left over from the calls before
    g.release()


@pytest.mark.parametrize("name", ["path7", "path8", "path9", "path40", "path41", "path1000", "grid", "uniform", "rmat"])
def test_levels(nwg, port, name):
    if name.startswith("path"):
        k = int(name[4:])
        u = np.arange(k - 1, dtype=np.uint64)
        off, cols = gg.csr_from_pairs(u, u + np.uint64(1), k)
    else:
        off, cols = {"grid": lambda: gg.grid(120, 70, 1, seed=1), "uniform": lambda: gg.uniform(20001, 9, seed=2),
                     "rmat": lambda: gg.rmat(14, 16, seed=3)}[name]()
    g = nwg.Graph.from_csr(off, cols)
    for r in map(int, gg.roots(off, 3, seed=4)):
        parents, _ = port.dobfs(off, cols, r)
        _same(nwg, port, g, off, cols, r, parents)
        bad = parents.copy()
        bad[int(np.flatnonzero(parents != NULL)[-1])] = NULL
        _same(nwg, port, g, off, cols, r, bad)
    g.release()
