"""Multi-source depth rows at every alignment: vertex counts around the
16-byte stores, the 512-vertex tiles and odd sizes, both row widths, arrays
that start off a 16-byte boundary.  Every value equals the oracle's and
nothing is written outside the rows."""
import numpy as np
import pytest

from oracle import graphgen as gg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 7, 15, 16, 17, 31, 33, 511, 512, 513, 1000, 1024, 1037, 5003])
def test_rows_at_every_alignment(nwg, port, n):
    import torch

    off, cols = gg.uniform(n, 3, seed=n)
    g = nwg.Graph.from_csr(off, cols)
    ws = nwg.MsWorkspace(g)
    for k in (1, 5, 65):
        roots = np.resize(gg.roots(off, min(k, 9), seed=k), k)
        want = port.msbfs_depths(off, cols, roots)
        for shift in range(0, 16, 3):
            buf = torch.full((k * n + 40,), 77, dtype=torch.uint8, device="cuda")
            ws.run_ex(roots, buf[shift:shift + k * n])
            h = buf.cpu().numpy()
            assert np.array_equal(h[shift:shift + k * n].reshape(k, n), want)
            assert np.all(h[:shift] == 77) and np.all(h[shift + k * n:] == 77)
        wide = np.where(want == 255, np.uint16(0xFFFF), want.astype(np.uint16))
        for shift in range(0, 8, 3):
            buf = torch.full((k * n + 20,), 7777, dtype=torch.int16, device="cuda")
            ws.run_ex(roots, buf[shift:shift + k * n])
            h = buf.cpu().numpy().view(np.uint16)
            assert np.array_equal(h[shift:shift + k * n].reshape(k, n), wide)
            assert np.all(h[:shift] == 7777) and np.all(h[shift + k * n:] == 7777)
    ws.close()
    g.release()
