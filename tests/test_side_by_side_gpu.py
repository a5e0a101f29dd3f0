"""Calls on one graph from two threads run side by side: while one thread is in
a long call, the other's short verifications and betweenness calls are
answered, exactly, again and again."""
import threading
import time

import numpy as np
import pytest

from oracle import graphgen as gg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("long_call", ["betweenness", "bfs_roots"])
@pytest.mark.parametrize("short_call", ["betweenness", "verify"])
def test_short_calls_beside_a_long_one(nwg, port, long_call, short_call):
    off, cols = gg.rmat(16, 16, seed=1)
    g = nwg.Graph.from_csr(off, cols)
    roots = gg.roots(off, 64, seed=2)
    r = int(roots[0])
    parents, _ = port.dobfs(off, cols, r)
    reached = np.count_nonzero(parents != 0xFFFFFFFF)
    alone, _ = nwg.betweenness(g, roots[:1])
    many = np.resize(roots, 2000).astype(np.uint32)
    rows = np.zeros((many.size, g.n), np.uint32)

    def long_one():
        if long_call == "betweenness":
            nwg.betweenness(g, many, lanes=1)
        else:
            nwg.bfs_roots(g, many, parents_out=rows)

    def short_one():
        if short_call == "betweenness":
            assert np.max(np.abs(nwg.betweenness(g, roots[:1])[0] - alone)) <= 1e-6
        else:
            res = nwg.verify(g, r, parents)
            assert res.valid == 1 and res.reached == reached

    nwg.bfs_roots(g, many[:4], parents_out=rows)
    short_one()
    started, failed = threading.Event(), []

    def run():
        started.set()
        try:
            long_one()
        except Exception as e:  # reported below, on the main thread
            failed.append(repr(e))

    t = threading.Thread(target=run)
    t.start()
    started.wait()
    time.sleep(0.005)
    answered = 0
    while t.is_alive():
        short_one()
        answered += t.is_alive()
    t.join()
    assert not failed, failed
    assert answered >= 5
    short_one()
    g.release()
