"""Device memory that graphs keep between calls: at most 2 GB over all graphs of
a device, and all of it given back when the graphs are released."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graphs(nwg, n, count, call="verify"):
    """`count` registrations of one graph of n vertices: the edges 0 <-> 1, or (many roots) a uniform graph of degree 16."""
    import torch

    if call == "bfs_roots":
        one = nwg.Graph.uniform(n, 16, seed=1)
        off, col = (torch.from_numpy(x.view(t)).cuda() for x, t in zip(one.csr(), (np.int64, np.int32)))
        one.release()
    else:
        off = torch.full((n + 1,), 2, dtype=torch.int64, device="cuda")
        off[0], off[1] = 0, 1
        col = torch.tensor([1, 0, 0, 0], dtype=torch.int32, device="cuda")[:2]
    return [nwg.Graph.from_csr(off, col, device=True) for _ in range(count)]


@pytest.mark.parametrize("call,n,count", [("verify", 1 << 24, 24), ("betweenness", 1 << 22, 8), ("bfs_roots", 1 << 17, 24)])
def test_kept_memory_is_bounded(nwg, call, n, count):
    import torch

    parents = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    parents[0] = parents[1] = 0
    rows = np.zeros((64, n), np.uint32) if call == "bfs_roots" else None

    def run(g):
        if call == "verify":
            assert nwg.verify(g, 0, parents).valid == 1
        elif call == "betweenness":
            scores, _ = nwg.betweenness(g, np.zeros(4, np.uint32), normalize=False, lanes=4)
            assert scores[0] == 4 and not scores[1:].any()
        else:
            nwg.bfs_roots(g, np.zeros(64, np.uint32), parents_out=rows)  # a block per root, 25 at once
            assert np.array_equal(rows != 0xFFFFFFFF, np.tile(nwg.bfs(g, root=0) != 0xFFFFFFFF, (64, 1)))

    graphs = _graphs(nwg, n, count, call)
    if call == "bfs_roots":  # the workspaces of nwg.bfs are not what is counted
        for g in graphs:
            nwg.bfs(g, root=0)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for g in graphs:
        run(g)
    kept = before - torch.cuda.mem_get_info()[0]
    assert kept <= (2 << 30) + (64 << 20)  # and what loading the kernels takes
    for g in graphs:  # kept states and others alike answer again
        run(g)
    for g in graphs:
        g.release()
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] <= 64 << 20
