"""Many roots of a small graph where the device has no room for their rows and
queues side by side (up to 128 MB): the traversals then run one after another
in the graph's workspaces, as they do on larger graphs."""
import numpy as np
import pytest

from oracle import graphgen as gg

pytestmark = pytest.mark.gpu


def test_roots_with_little_memory_left(nwg, port):
    import torch

    off, cols = gg.uniform(1 << 17, 16, seed=1)
    g = nwg.Graph.from_csr(off, cols)
    roots = gg.roots(off, 64, seed=2)
    small = nwg.Graph.from_csr(*gg.uniform(20000, 16, seed=3))
    nwg.bfs_roots(small, small.roots(64))  # the kernels of both ways are loaded
    nwg.bfs(g, root=int(roots[0]))
    rows = np.empty((roots.size, g.n), np.uint32)
    torch.cuda.synchronize()
    room = torch.cuda.mem_get_info()[0] - (72 << 20)
    held = torch.empty(room, dtype=torch.uint8, device="cuda")
    try:
        left = torch.cuda.mem_get_info()[0]
        assert left < 100 << 20  # less than the rows and queues take
        status = np.full(roots.size, -7, np.int32)
        nwg.bfs_roots(g, roots, parents_out=rows, status=status)
    finally:
        del held
        torch.cuda.empty_cache()
    assert np.all(status == 0)
    for i in range(0, roots.size, 9):
        r = int(roots[i])
        assert np.array_equal(nwg.depths_from_parents(rows[i], r), port.depths(off, cols, r))
    again = nwg.bfs_roots(g, roots)  # and side by side again
    for i in range(0, roots.size, 9):
        assert port.verify(off, cols, int(roots[i]), again[i])
    g.release()
    small.release()
