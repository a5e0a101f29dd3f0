"""The device verifier's state: levels whose pieces do not fit its queues of
n / 4 + m / 512 entries (pulled, or on a graph whose in-CSR is not the
transpose pushed from their depths), against the reference's verdicts
(restated in test_verify_gpu.py), and the memory that a graph keeps after a
verification, within the 12 bytes a vertex that the depths and two queues of
vertices would take."""
import numpy as np
import pytest

from oracle import graphgen as gg
from test_verify_gpu import reference_verdict

pytestmark = pytest.mark.gpu
NULL = 0xFFFFFFFF


def _wide(mids, dense, both):
    """Root 0 - mids - a leaf each, beside a complete graph: a level of many vertices with few of the graph's edges."""
    mid = np.arange(1, mids + 1, dtype=np.uint64)
    x, y = (t.astype(np.uint64) + np.uint64(2 * mids + 1) for t in np.triu_indices(dense, 1))
    u = np.concatenate([np.zeros(mids, np.uint64), mid, x])
    v = np.concatenate([mid, mid + np.uint64(mids), y])
    n = 2 * mids + 1 + dense
    return gg.csr_from_pairs(u, v, n) if both else gg.directed_csr(u, v, n)


@pytest.mark.parametrize("mids,dense", [(3000, 300), (40000, 900), (1, 3), (31, 40)])
@pytest.mark.parametrize("both", [True, False])
def test_levels_that_do_not_fit(nwg, port, mids, dense, both):
    off, cols = _wide(mids, dense, both)
    n = off.size - 1
    if mids >= 3000:  # the middle level has a piece for each vertex
        assert mids > n // 4 + cols.size // 512 + 1
    g = nwg.Graph.from_csr(off, cols)
    for root in (0, 1, n - 2):
        parents, _ = port.dobfs(off, cols, root, *gg.transpose(off, cols, n))
        bad = parents.copy()
        bad[int(np.flatnonzero(parents != NULL)[-1])] = NULL
        for p in (parents, bad):
            want = reference_verdict(port, off, cols, root, p)
            got = nwg.verify(g, root, p)
            assert bool(got.valid) == want[0]
            if not want[0]:
                assert (got.first_bad, got.reason) == (want[1], want[2])
            depth = port.depths(off, cols, root)
            assert got.reached == np.count_nonzero(depth != NULL)
            assert got.levels == depth[depth != NULL].max() + 1
    g.release()


def test_memory_of_a_verification(nwg):
    import torch

    n = 1 << 24
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = 1  # one edge, 0 -> 0
    col = torch.zeros(4, dtype=torch.int32, device="cuda")
    parents = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    parents[0] = 0
    g = nwg.Graph.from_csr(off, col[:1], device=True)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    res = nwg.verify(g, 0, parents)
    assert res.valid == 1 and res.reached == 1 and res.levels == 1
    assert before - torch.cuda.mem_get_info()[0] <= 12 * n
    g.release()
