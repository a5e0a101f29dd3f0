"""nwg.verify on a device tensor that work queued on torch's current stream still
writes: the check reads what that work leaves."""
import pytest

from oracle import graphgen as gg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [False, True])
def test_verify_reads_what_the_current_stream_writes(nwg, port, side):
    import torch

    off, cols = gg.rmat(12, 16, seed=1)
    g = nwg.Graph.from_csr(off, cols)
    r = int(gg.roots(off, 1, seed=2)[0])
    good = torch.from_numpy(port.dobfs(off, cols, r)[0].view("int32")).cuda()
    parents = torch.empty_like(good)
    assert nwg.verify(g, r, good).valid == 1  # the graph's state is made
    torch.cuda.synchronize()
    stream = torch.cuda.Stream() if side else torch.cuda.current_stream()
    with torch.cuda.stream(stream):
        for start, end, valid in ((-1, good, 1), (good, -1, 0)):
            parents.copy_(start) if torch.is_tensor(start) else parents.fill_(start)
            torch.cuda.synchronize()
            torch.cuda._sleep(100_000_000)  # about 50 ms, then the write
            parents.copy_(end) if torch.is_tensor(end) else parents.fill_(end)
            assert nwg.verify(g, r, parents).valid == valid
    g.release()
