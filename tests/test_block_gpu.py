"""One-block traversals (bitmaps in shared memory): single traversals of small
graphs, many roots of a graph, ragged batches.  Depths bit-exact with the
oracle, parents within BFSVerifier's rules, directions and discoveries per
step equal to the restatement's, at the sizes where the block path changes:
words that are not full, the queue in shared or device memory (2,048
vertices), more hubs than a step lists, the last graph it takes and the first
it does not."""
import numpy as np
import pytest

from oracle import graphgen as gg

pytestmark = pytest.mark.gpu
NULL = 0xFFFFFFFF


def _hubs(k, deg):
    """Root 0 joined to k hubs, each joined to `deg` leaves of its own."""
    u = np.concatenate([np.zeros(k, np.uint64), np.repeat(np.arange(1, k + 1, dtype=np.uint64), deg)])
    v = np.concatenate([np.arange(1, k + 1, dtype=np.uint64), np.arange(k + 1, k + 1 + k * deg, dtype=np.uint64)])
    return gg.csr_from_pairs(u, v, 1 + k + k * deg)


GRAPHS = {
    "two": lambda: gg.csr_from_pairs(np.array([0], np.uint64), np.array([1], np.uint64), 2),
    "n31": lambda: gg.uniform(31, 4, seed=1),
    "n33": lambda: gg.uniform(33, 4, seed=2),
    "n2048": lambda: gg.uniform(2048, 8, seed=3),
    "n2049": lambda: gg.uniform(2049, 8, seed=4),
    "star600": lambda: gg.csr_from_pairs(np.zeros(600, np.uint64), np.arange(1, 601, dtype=np.uint64), 601),
    "hubs140": lambda: _hubs(140, 600),  # 84,141 vertices: k_trav; its roots go to blocks
    "hubs20": lambda: _hubs(20, 600),
    "limit": lambda: gg.uniform(1 << 15, 6, seed=5),
    "past_limit": lambda: gg.uniform((1 << 15) + 1, 6, seed=6),
}


def _check(port, nwg, off, cols, root, parents, in_off=None, in_cols=None):
    want = port.depths(off, cols, root)
    assert np.array_equal(nwg.depths_from_parents(parents, root), want)
    assert np.array_equal(parents != NULL, want != NULL)
    assert port.verify(off, cols, root, parents, in_off, in_cols)


@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_block_traversals(nwg, port, name):
    import torch

    off, cols = GRAPHS[name]()
    g = nwg.Graph.from_csr(off, cols)
    n = g.n
    roots = np.unique(np.concatenate([gg.roots(off, 3, seed=7), [0, n - 1]])).astype(np.uint32)
    for r in map(int, roots):
        for alpha, beta in ((15, 18), (1, 1), (1000000, 18)):
            parents, st = nwg.bfs(g, g, r, 32, alpha, beta, stats=True)
            _check(port, nwg, off, cols, r, parents)
            _, tr = port.dobfs(off, cols, r, alpha=alpha, beta=beta)
            got = st.trace()
            for key in ("dir", "found", "frontier"):
                assert np.array_equal(got[key], np.asarray(tr[key])[: got[key].size]), key
            assert got["dir"].size == len(tr["dir"]) and st.status == 0
        _check(port, nwg, off, cols, r, nwg.bfs_serial(g, r))
    # a parents array that starts at any 4-byte boundary
    r = int(roots[0])
    for shift in (1, 2, 3):
        buf = torch.full((n + 8,), 7, dtype=torch.int32, device="cuda")
        nwg.bfs_device(g, r, buf[shift:shift + n])
        host = buf.cpu().numpy().view(np.uint32)
        _check(port, nwg, off, cols, r, host[shift:shift + n])
        assert np.all(host[:shift] == 7) and np.all(host[shift + n:] == 7)
    # many roots: odd counts, repeats
    many = np.resize(roots, 2 * roots.size + 1)
    status = np.full(many.size, -7, np.int32)
    rows = nwg.bfs_roots(g, many, status=status)
    assert np.all(status == 0)
    for i, x in enumerate(many):
        _check(port, nwg, off, cols, int(x), rows[i])
    g.release()


def test_block_roots_over_several_chunks_directed(nwg, port):
    """More roots than a launch takes (chunks of at most two blocks per SM,
    fewer on the larger graph), on a directed pair."""
    rng = np.random.default_rng(2)
    for n, m, k in ((3000, 12000, 700), (120000, 500000, 120)):
        u, v = (rng.integers(0, n, m).astype(np.uint64) for _ in range(2))
        off, cols = gg.directed_csr(u, v, n)
        in_off, in_cols = gg.transpose(off, cols, n)
        g = nwg.Graph.from_csr(off, cols, in_off, in_cols)
        roots = gg.roots(off, k, seed=9)
        rows = nwg.bfs_roots(g, roots)
        for i in list(range(0, k, max(1, k // 12))) + [k - 1]:
            _check(port, nwg, off, cols, int(roots[i]), rows[i], in_off, in_cols)
        again = nwg.bfs_roots(g, roots[:5])
        for i in range(5):
            _check(port, nwg, off, cols, int(roots[i]), again[i], in_off, in_cols)
        g.release()


def test_ragged_mixes_queue_places_and_a_large_graph(nwg, port):
    """Queues in shared and in device memory in one launch, and a graph past
    the block path's 2^19 vertices, whose items keep the block-per-item
    kernel with its state in device memory."""
    graphs = [gg.uniform(2048, 6, seed=1), gg.grid(60, 50, 1, seed=2), gg.rmat(13, 8, seed=3), gg.uniform(50, 3, seed=4),
              gg.uniform((1 << 19) + 5, 3, seed=5)]
    for chosen in (graphs, graphs[:4]):
        batch = nwg.RaggedBatch(chosen)
        items = [(gi, int(r), 15, 18, 32) for gi, (off, _) in enumerate(chosen) for r in gg.roots(off, 2, seed=gi)]
        for bps in (1, 2):
            parents, offs, res, _ = batch.run(items, blocks_per_sm=bps)
            host = parents.cpu().numpy().view(np.uint32)
            for i, (gi, r, *_rest) in enumerate(items):
                off, cols = chosen[gi]
                _check(port, nwg, off, cols, r, host[offs[i]:offs[i] + off.size - 1])
                assert res[i].status == 0 and res[i].reached == np.count_nonzero(port.depths(off, cols, r) != NULL)
        batch.release()


@pytest.mark.parametrize("n,deg", [(1500, 8), (2100, 8), (40000, 8)])
def test_noalloc_block_and_grid(nwg, port, n, deg):
    import torch

    off, cols = gg.uniform(n, deg, seed=n)
    dev = [torch.from_numpy(off.view(np.int64)).cuda(), torch.from_numpy(cols.view(np.int32)).cuda()]
    par = torch.empty(n, dtype=torch.int32, device="cuda")
    for r in map(int, gg.roots(off, 3, seed=1)):
        nwg.bfs_noalloc(*dev, n, r, par)
        _check(port, nwg, off, cols, r, par.cpu().numpy().view(np.uint32))
