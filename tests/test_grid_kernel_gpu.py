"""The whole-grid traversal kernel on what small graphs exercise: the graphs of
the solo-level, directed, parameter, golden and thread tests with 40,000
isolated vertices behind them and all their other ids kept, so that they are
past the one-block sizes.  Depths, parents and per-step traces equal the
oracle's, the trace whole (up to its 256 records)."""
import threading

import numpy as np
import pytest

from oracle import graphgen as gg
from test_dobfs_gpu import _fan_bipartite, _path_star
from test_pull_batch_gpu import _sparse

pytestmark = pytest.mark.gpu
NULL = 0xFFFFFFFF
BEHIND = 40000


def _behind(off, cols):
    """The CSR with BEHIND isolated vertices after its own."""
    off = np.asarray(off, np.uint64)
    return np.concatenate([off, np.full(BEHIND, off[-1])]), np.asarray(cols, np.uint32)


def _check(nwg, port, g, csr, r, alpha=15, beta=18, topdown=False):
    off, cols = csr[:2]
    parents, st = nwg.bfs_serial(g, r, stats=True) if topdown else nwg.bfs(g, g, r, 32, alpha, beta, stats=True)
    want = port.depths(off, cols, r)
    assert np.array_equal(nwg.depths_from_parents(parents, r), want)
    assert port.verify(off, cols, r, parents, *csr[2:])
    assert st.status == 0 and st.kernel_launches == 1
    got = st.trace()
    if topdown:
        assert not got["dir"].any()
        return st
    _, tr = port.dobfs(off, cols, r, *csr[2:], alpha=alpha, beta=beta)
    m = got["dir"].size
    assert m == min(len(tr["dir"]), 256)
    for key in ("dir", "found", "frontier"):
        assert np.array_equal(got[key], np.asarray(tr[key])[:m]), key
    return st


def test_solo_levels_on_the_grid(nwg, port):
    u = np.arange(1999, dtype=np.uint64)
    for csr, roots in ((gg.csr_from_pairs(u, u + np.uint64(1), 2000), (0, 777, 1999)),
                       (_path_star(40, 20000, 3), (0, 20, 39, 40 + 123)), (_path_star(300, 6000, 9), (0, 150))):
        csr = _behind(*csr)
        g = nwg.Graph.from_csr(*csr)
        for r in roots:
            _check(nwg, port, g, csr, r)
            _check(nwg, port, g, csr, r, topdown=True)
        g.release()


@pytest.mark.parametrize("alpha,beta", [(15, 18), (1, 1), (1000000, 18), (15, 1000000), (100, 1000)])
def test_parameters_on_the_grid(nwg, port, alpha, beta):
    for csr in (gg.rmat(13, 16, seed=7), gg.uniform(9000, 10, seed=8), gg.grid(70, 60, 1, seed=9), _fan_bipartite(n2=4096)):
        csr = _behind(*csr)
        g = nwg.Graph.from_csr(*csr)
        for r in map(int, gg.roots(csr[0], 3, seed=4)):
            _check(nwg, port, g, csr, r, alpha, beta)
        g.release()


def test_directed_pairs_on_the_grid(nwg, port):
    rng = np.random.default_rng(11)
    for n, m in ((3000, 20000), (2000, 200000), (20000, 50000)):
        off, cols = gg.directed_csr(*(rng.integers(0, n, m).astype(np.uint64) for _ in range(2)), n)
        csr = (*_behind(off, cols), *_behind(*gg.transpose(off, cols, n)))
        g = nwg.Graph.from_csr(*csr)
        for r in map(int, gg.roots(off, 4, seed=12)):
            _check(nwg, port, g, csr, r)
            _check(nwg, port, g, csr, r, 1000000, 1)
        g.release()


def test_golden_graphs_on_the_grid(nwg, port, golden):
    for G in golden:
        csr = _behind(G.off, G.cols)
        if G.in_off is not None:
            csr = (*csr, *_behind(G.in_off, G.in_cols))
        g = nwg.Graph.from_csr(*csr)
        for i, r in enumerate(map(int, G.roots)):
            parents = nwg.bfs(g, root=r)
            assert np.array_equal(nwg.depths_from_parents(parents, r)[: G.n], G.depths[i])
            assert np.all(parents[G.n:] == NULL)
        g.release()


def test_grids_beside_one_another_from_threads(nwg, port):
    import torch

    u = np.arange(2999, dtype=np.uint64)
    hosts = [_behind(*gg.csr_from_pairs(u, u + np.uint64(1), 3000)), _behind(*gg.rmat(14, 16, seed=4))]
    graphs = [nwg.Graph.from_csr(*h) for h in hosts]
    jobs = [(0, 0), (0, 1500)] + [(1, int(r)) for r in gg.roots(hosts[1][0], 2, seed=8)]
    want = {(i, r): port.depths(*hosts[i], r) for i, r in jobs}
    errors = []

    def worker(order):
        try:
            stream = torch.cuda.Stream()
            wss = [g.workspace() for g in graphs]
            outs = [torch.empty(g.n, dtype=torch.int32, device="cuda") for g in graphs]
            for i, r in order * 4:
                wss[i].bfs_async(r, outs[i], stream.cuda_stream)
                stream.synchronize()
                p = outs[i].cpu().numpy().view(np.uint32)
                if wss[i].stats().status != 0 or not np.array_equal(nwg.depths_from_parents(p, r), want[(i, r)]):
                    errors.append((i, r, wss[i].stats().status))
            for w in wss:
                w.close()
        except Exception as e:  # reported below, on the main thread
            errors.append(repr(e))

    threads = [threading.Thread(target=worker, args=(j,)) for j in (jobs, jobs[::-1])]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for g in graphs:
        g.release()
    assert not errors, errors[:5]


@pytest.mark.parametrize("n,deg,directed", [(32769, 32, False), (40000, 14, False), (49999, 37, False), (90001, 45, False),
                                            (100003, 20, False), (131073, 51, False), (32769, 64, True), (49999, 74, True)])
def test_offering_steps_run(nwg, port, n, deg, directed):
    """Uniform graphs with a step of n / 2 to 2.5 n front edges (a power of the
    degree), which offers parents; parents arrays at any 4-byte boundary."""
    import torch

    off, cols = gg.uniform(n, deg, seed=n + deg)
    csr = (off, cols)
    if directed:  # every other arc
        src = np.repeat(np.arange(n, dtype=np.uint64), np.diff(off).astype(np.int64))
        csr = gg.directed_csr(src[::2], cols[::2].astype(np.uint64), n)
        csr = (*csr, *gg.transpose(*csr, n))
    g = nwg.Graph.from_csr(*csr)
    offers = 0
    for i, r in enumerate(map(int, gg.roots(off, 3, seed=deg))):
        offers += _check(nwg, port, g, csr, r).offer_steps
        buf = torch.full((n + 8,), 7, dtype=torch.int32, device="cuda")
        offers += nwg.bfs_device(g, r, buf[i + 1:i + 1 + n], stats=True).offer_steps
        host = buf.cpu().numpy().view(np.uint32)
        assert port.verify(*csr[:2], r, host[i + 1:i + 1 + n], *csr[2:])
        assert np.all(host[: i + 1] == 7) and np.all(host[i + 1 + n:] == 7)
    assert offers >= 2
    g.release()


@pytest.mark.parametrize("n,deg,directed", [(40000, 4, False), (65535, 4, True), (131072, 2, False)])
def test_traces_of_sparse_pulls_are_whole(nwg, port, n, deg, directed):
    csr = _sparse(n, deg, n // 2000, n, directed)
    csr = csr[: 4 if directed else 2]
    g = nwg.Graph.from_csr(*csr)
    assert sum(_check(nwg, port, g, csr, r, *ab).bu_steps for r in map(int, gg.roots(csr[0], 3, seed=deg))
               for ab in ((15, 18), (100, 1000))) > 0
    g.release()


def test_hubs_do_not_offer(nwg, port):
    off, cols = gg.rmat(16, 16, seed=1)
    g = nwg.Graph.from_csr(off, cols)
    for r in map(int, gg.roots(off, 3, seed=2)):
        assert _check(nwg, port, g, (off, cols), r).offer_steps == 0
    g.release()


def _hubs(k, leaves):
    """Root 0 joined to k hubs, each joined to the same leaves."""
    hub = np.arange(1, k + 1, dtype=np.uint64)
    leaf = np.arange(k + 1, k + 1 + leaves, dtype=np.uint64)
    u = np.concatenate([np.zeros(k, np.uint64), np.repeat(hub, leaves)])
    return gg.csr_from_pairs(u, np.concatenate([hub, np.tile(leaf, k)]), k + 1 + leaves)


@pytest.mark.parametrize("k", [127, 128, 129, 140])
def test_more_hubs_than_a_block_lists(nwg, port, k):
    """A one-block step lists at most 128 vertices of more than 512 out-edges;
    further ones stay with their warp: in a single traversal, in a batch's
    items and in many roots side by side (alpha 1 keeps the hubs' step a push)."""
    off, cols = _hubs(k, 600)
    other = gg.uniform(500, 6, seed=1)
    g = nwg.Graph.from_csr(off, cols)
    parents, st = nwg.bfs(g, g, 0, 32, 1, 18, stats=True)
    assert list(st.trace()["dir"][:2]) == [0, 0] and st.trace()["found"][1] == 600
    rows = nwg.bfs_roots(g, np.zeros(40, np.uint32), alpha=1)
    batch = nwg.RaggedBatch([(off, cols), other])
    packed, offs, res, _ = batch.run([(1, 3, 15, 18, 32), (0, 0, 1, 18, 32), (0, 0, 15, 18, 32)])
    packed = packed.cpu().numpy().view(np.uint32)
    want = port.depths(off, cols, 0)
    for p in (parents, rows[0], rows[39], *(packed[int(offs[i]):int(offs[i]) + g.n] for i in (1, 2))):
        assert np.array_equal(nwg.depths_from_parents(p, 0), want)
        assert port.verify(off, cols, 0, p)
    assert res[1].td_steps >= 2 and res[1].reached == g.n
    batch.release()
    g.release()
