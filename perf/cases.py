"""The workloads this library is timed on: one dict per case, sizes from bench.py and the tests.

listed() names the standing cases, draw(rng) gives further ones of the same
ranges, prepare(case, seed) builds what a program holds before the call,
run(state) makes the call, work(case) counts the bytes it cannot do without
and exact(case, seed) gives floating results in 64 bits.

Graphs are made with torch from the seed and registered as device arrays (or
uploaded from the host where the case says so).  Which front vertex becomes a
parent is a race in a top-down step, so a traversal's parents are returned as
the reached set (a bool per vertex) with the vertices found at every step.
"""
import math

import numpy as np
import torch

import nwgr_b200 as nwg

A, AB, ABC = 0.57, 0.76, 0.95  # cumulative RMAT quadrant probabilities (Graph500)


def listed():
    return [
        # Graph500 / GAP-Kron style traversal, the headline workload: hubs, 8-9 steps
        {"name": "bfs_rmat24", "op": "bfs", "kind": "rmat", "n": 1 << 24, "degree": 32, "roots": 4},
        # GAP-Urand style: no hubs, the discovering step is most of the time
        {"name": "bfs_uniform24", "op": "bfs", "kind": "uniform", "n": 1 << 24, "degree": 32, "roots": 2},
        # road-like mesh with shortcuts: many thin levels
        {"name": "bfs_grid4096", "op": "bfs", "kind": "grid", "n": 1 << 24, "degree": 4, "roots": 2},
        # the drop-in call on a small graph: latency, parents to the host
        {"name": "bfs_rmat10_host", "op": "bfs_host", "kind": "rmat", "n": 1 << 10, "degree": 32, "topdown": False},
        # a latency-bound service that may not allocate, its own device arrays
        {"name": "noalloc_rmat16", "op": "noalloc", "kind": "rmat", "n": 1 << 16, "degree": 32},
        # the benchmark loop over many sources: directed pair, 32-bit offsets, odd size, parents to pinned host rows
        {"name": "roots_directed", "op": "roots", "kind": "uniform", "n": 20011, "degree": 5, "roots": 64},
        # 64 sources in one word (all-pairs distance sampling, landmarks)
        {"name": "msbfs64_rmat22", "op": "msbfs", "kind": "rmat", "n": 1 << 22, "degree": 32, "roots": 64, "width": 1},
        # an odd source count on an odd uniform graph, 16-bit rows
        {"name": "msbfs100_u16", "op": "msbfs", "kind": "uniform", "n": 1000003, "degree": 16, "roots": 100, "width": 2},
        # many small graphs of mixed shapes and sizes in one launch
        {"name": "ragged_256", "op": "ragged", "graphs": 256, "roots": 4, "lo": 10, "hi": 18},
        # a burst of (graph, root) queries to the server, answers in host rows
        {"name": "serve_burst", "op": "serve", "graphs": 32, "queries": 2000, "lo": 10, "hi": 16, "width": 1},
        # checking a traversal's parents on the device
        {"name": "verify_rmat22", "op": "verify", "kind": "rmat", "n": 1 << 22, "degree": 32, "host": False},
        # approximate betweenness centrality over a few sources
        {"name": "bc_rmat20", "op": "bc", "kind": "rmat", "n": 1 << 20, "degree": 32, "roots": 8},
    ]


def _log(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["bfs", "bfs", "bfs", "bfs_host", "noalloc", "roots", "msbfs", "msbfs", "ragged", "serve", "verify", "bc"])
    kind = rng.choice(["rmat", "uniform", "grid"])
    degree = 4 if kind == "grid" else 2 * _log(rng, 4, 16)
    if op == "bfs":
        return {"op": op, "kind": kind, "n": _log(rng, 1 << 16, 1 << 24), "degree": degree, "roots": rng.randint(1, 4)}
    if op == "bfs_host":
        return {"op": op, "kind": kind, "n": _log(rng, 200, 1 << 17), "degree": degree, "topdown": rng.random() < 0.4}
    if op in ("noalloc", "verify") and kind != "rmat":  # sparse ones, with vertices out of reach
        kind, degree = "uniform", 4
    if op == "noalloc":
        return {"op": op, "kind": kind, "n": _log(rng, 1 << 10, 1 << 18), "degree": degree}
    if op == "roots":
        kind = rng.choice(["rmat", "uniform"])
        return {"op": op, "kind": kind, "n": _log(rng, 1 << 12, 1 << 17), "degree": rng.randint(2, 6), "roots": rng.randint(8, 64)}
    if op == "msbfs":
        kind = rng.choice(["rmat", "uniform"])
        return {"op": op, "kind": kind, "n": _log(rng, 1 << 14, 1 << 21), "degree": 2 * _log(rng, 4, 16),
                "roots": _log(rng, 1, 300), "width": rng.choice([1, 2])}
    if op == "ragged":
        return {"op": op, "graphs": _log(rng, 32, 256), "roots": rng.randint(1, 4), "lo": 10, "hi": rng.randint(14, 18)}
    if op == "serve":
        return {"op": op, "graphs": _log(rng, 8, 32), "queries": _log(rng, 200, 2000), "lo": 10, "hi": rng.randint(13, 16),
                "width": rng.choice([1, 2])}
    if op == "verify":
        return {"op": op, "kind": kind, "n": _log(rng, 1 << 12, 1 << 22), "degree": degree, "host": rng.random() < 0.3}
    return {"op": op, "kind": kind, "n": _log(rng, 1 << 12, 1 << 20 if kind != "grid" else 1 << 16), "degree": degree,
            "roots": rng.randint(1, 8)}


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _arcs(case, gen, arcs):
    """`arcs` random arcs (source, target) of the case's family; a grid's are its right and down neighbours and 1% shortcuts."""
    n = case["n"]
    if case["kind"] == "uniform":
        return torch.randint(0, n, (arcs,), generator=gen, device="cuda"), torch.randint(0, n, (arcs,), generator=gen, device="cuda")
    if case["kind"] == "grid":
        w = max(2, math.isqrt(n))
        v = torch.arange(n, device="cuda")
        right, down = v[(v % w != w - 1) & (v + 1 < n)], v[v + w < n]
        a, b = (torch.randint(0, n, (n // 100,), generator=gen, device="cuda") for _ in range(2))
        return torch.cat([right, down, a]), torch.cat([right + 1, down + w, b])
    scale = max(1, (n - 1).bit_length())
    u = torch.zeros(arcs, dtype=torch.int32, device="cuda")
    v = torch.zeros(arcs, dtype=torch.int32, device="cuda")
    for _ in range(scale):
        r = torch.rand(arcs, generator=gen, device="cuda")
        u.mul_(2).add_(r >= AB)
        v.mul_(2).add_(((r >= A) & (r < AB)) | (r >= ABC))
    perm = torch.randperm(1 << scale, generator=gen, device="cuda")
    return perm[u] % n, perm[v] % n


def _csr(src, dst, n):
    """Sorted rows without duplicates: offsets (int64) and columns (int32)."""
    key = (src * n).add_(dst)
    key = torch.unique_consecutive(torch.sort(key).values)
    off = torch.searchsorted(key, torch.arange(n + 1, device="cuda") * n)
    return off, (key % n).to(torch.int32)


def _graph(case, gen):
    """Symmetric CSR without self-loops."""
    n = case["n"]
    u, v = _arcs(case, gen, n * case["degree"] // 2)
    keep = u != v
    u, v = u[keep], v[keep]
    return _csr(torch.cat([u, v]), torch.cat([v, u]), n)


def _pick(off, count, gen):
    """`count` random vertices with out-edges."""
    c = torch.randint(0, off.numel() - 1, (64 * count + 4096,), generator=gen, device="cuda")
    return c[off[c + 1] > off[c]][:count].cpu().numpy().astype(np.uint32)


def _parents(off, col, n, root):
    """A BFS tree: every reached vertex's parent is its first in-neighbour one level closer."""
    src = torch.repeat_interleave(torch.arange(n, device="cuda"), off[1:] - off[:-1])
    parent = torch.full((n,), n, dtype=torch.int64, device="cuda")
    front = torch.zeros(n, dtype=torch.bool, device="cuda")
    parent[root], front[root] = root, True
    while True:
        e = front[src] & (parent[col] == n)
        if not bool(e.any()):
            break
        t = col[e].long()
        parent.scatter_reduce_(0, t, src[e], "amin")
        front.zero_()
        front[t] = True
    return torch.where(parent == n, -1, parent).to(torch.int32)


def _many(case, seed):
    """Host CSRs of many graphs, half RMAT and half grids as in the ragged benchmark, and roots of each: sizes by the case, edges and roots by the seed."""
    rng = np.random.default_rng(case["graphs"])
    graphs, roots = [], []
    for i in range(case["graphs"]):
        size, ef = rng.uniform(case["lo"], case["hi"]), int(rng.integers(8, 33))
        if i % 2 == 0:
            g = nwg.Graph.rmat(round(size), ef, seed=seed * 1009 + i)
        else:
            w = max(2, round(2 ** (size / 2)))
            g = nwg.Graph.grid(w, max(2, int(2**size) // w), 1, seed=seed * 1009 + i)
        graphs.append(g.csr())
        roots.append(g.roots(4, seed=seed * 7919 + i))
        g.release()
    return graphs, roots


def prepare(case, seed):
    op, gen = case["op"], _generator(seed)
    s = {"op": op, "case": case}
    if op in ("ragged", "serve"):
        hosts, roots = _many(case, seed)
        sizes = [off.size - 1 for off, _ in hosts]
        if op == "ragged":
            s["batch"] = nwg.RaggedBatch(hosts)
            s["items"] = [(g, int(r), 15, 18, 32) for g in range(len(hosts)) for r in roots[g][: case["roots"]]]
            s["out"] = torch.empty(sum(sizes) * case["roots"], dtype=torch.int32, device="cuda")
            return s
        s["server"] = nwg.Server([nwg.Graph.from_csr(o, c) for o, c in hosts], slots=16, depth_bytes=case["width"])
        q = case["queries"]
        p = 1.0 / np.arange(1, len(hosts) + 1) ** 1.1  # popularity
        s["graph"] = np.random.default_rng(q).choice(len(hosts), q, p=p / p.sum()).astype(np.uint32)
        s["root"] = np.array([roots[g][i % 4] for i, g in enumerate(s["graph"])], np.uint32)
        s["arrival"] = np.zeros(q)
        ends = np.cumsum([sizes[g] for g in s["graph"]])
        s["buffer"] = np.zeros(ends[-1], np.uint8 if case["width"] == 1 else np.uint16)
        s["rows"] = [s["buffer"][e - sizes[g]:e] for e, g in zip(ends.tolist(), s["graph"])]
        return s
    n = case["n"]
    if op == "roots":  # a directed pair with 32-bit offsets, from the host
        u, v = _arcs(case, gen, n * case["degree"])
        out_csr, in_csr = _csr(u, v, n), _csr(v, u, n)
        host = [x.cpu().numpy().astype(np.uint32) for x in (*out_csr, *in_csr)]
        s["graph"] = nwg.Graph.from_csr(*host)
        s["roots"] = _pick(out_csr[0], case["roots"], gen)
        s["rows"] = torch.empty((case["roots"], n), dtype=torch.int32, pin_memory=True).numpy()
        return s
    off, col = _graph(case, gen)
    roots = _pick(off, case.get("roots", 1), gen)
    s["roots"] = [int(r) for r in roots]
    if op == "noalloc":
        s["off"], s["col"], s["parents"] = off, col, torch.empty(n, dtype=torch.int32, device="cuda")
        return s
    s["graph"] = nwg.Graph.from_csr(off, col, device=True)
    if op == "bfs":
        s["ws"] = s["graph"].workspace()
        s["parents"] = torch.empty(n, dtype=torch.int32, device="cuda")
    elif op == "bfs_host":
        s["parents"] = np.empty(n, np.uint32)
    elif op == "msbfs":
        s["roots"] = roots
        s["ws"] = nwg.MsWorkspace(s["graph"])
        s["depths"] = torch.empty((roots.size, n), dtype=torch.uint8 if case["width"] == 1 else torch.int16, device="cuda")
    elif op == "verify":
        s["parents"] = _parents(off, col, n, s["roots"][0])
        if case["host"]:
            s["parents"] = s["parents"].cpu().numpy().view(np.uint32)
    return s


def run(s):
    op, case = s["op"], s["case"]
    if op == "bfs":
        out = []
        for root in s["roots"]:
            s["ws"].bfs_async(root, s["parents"])  # in torch's stream order
            reached = s["parents"] != -1
            st = s["ws"].stats()
            out.append({"reached": reached, "levels": st.levels, "found": np.array(st.trace_found, np.int64)})
        return out
    if op == "bfs_host":
        if case["topdown"]:
            parents, st = nwg.bfs_serial(s["graph"], s["roots"][0], stats=True)
        else:
            parents, st = nwg.bfs(s["graph"], root=s["roots"][0], parents_out=s["parents"], stats=True)
        return {"reached": parents != nwg.NULL_VERTEX, "levels": st.levels, "found": np.array(st.trace_found[:16], np.int64)}
    if op == "noalloc":
        nwg.bfs_noalloc(s["off"], s["col"], case["n"], s["roots"][0], s["parents"])
        return s["parents"] != -1
    if op == "roots":
        return nwg.bfs_roots(s["graph"], s["roots"], parents_out=s["rows"]) != -1
    if op == "msbfs":
        st = s["ws"].run_ex(s["roots"], s["depths"])
        return {"depths": s["depths"], "levels": st.levels}
    if op == "ragged":
        torch.cuda.current_stream().synchronize()  # the batch has a stream of its own: the buffer's last reader first
        parents, offsets, results, _ = s["batch"].run(s["items"], s["out"])
        return {"reached": parents != -1, "offsets": offsets.astype(np.int64), "levels": np.array([r.levels for r in results], np.int64)}
    if op == "serve":
        s["server"].run_trace(s["graph"], s["root"], s["arrival"], s["rows"])
        return s["buffer"]
    if op == "verify":
        r = nwg.verify(s["graph"], s["roots"][0], s["parents"])
        return [r.valid, r.reason, r.reached, r.levels]
    scores, st = nwg.betweenness(s["graph"], s["roots"])
    return {"scores": scores, "levels": st.max_levels}


def work(case):
    """Every adjacency entry and offset read once, every result written once."""
    op = case["op"]
    if op in ("ragged", "serve"):
        per = (2.0 ** case["hi"] - 2.0 ** case["lo"]) / (math.log(2) * (case["hi"] - case["lo"]))  # mean vertices of a graph
        if op == "ragged":
            return {"bytes": case["graphs"] * case["roots"] * per * (4 * 22 + 12), "flops": 0}
        return {"bytes": case["graphs"] * per * (4 * 22 + 8) + case["queries"] * per * case["width"], "flops": 0}
    n, edges = case["n"], case["n"] * case["degree"]
    graph = 4 * edges + 8 * n
    if op == "bfs":
        return {"bytes": case["roots"] * (graph + 4 * n), "flops": 0}
    if op == "roots":
        return {"bytes": case["roots"] * (graph + 4 * n), "flops": 0}
    if op == "msbfs":
        return {"bytes": -(-case["roots"] // 256) * graph + case["roots"] * n * case["width"], "flops": 0}
    if op == "bc":
        return {"bytes": case["roots"] * (2 * graph + 16 * n), "flops": case["roots"] * 4.0 * edges}
    return {"bytes": graph + 4 * n, "flops": 0}


def exact(case, seed):
    """Brandes in 64 bits with plain torch; the other cases' results are whole numbers."""
    if case["op"] != "bc":
        return None
    n, gen = case["n"], _generator(seed)
    off, col = _graph(case, gen)
    roots = _pick(off, case["roots"], gen)
    src = torch.repeat_interleave(torch.arange(n, device="cuda"), off[1:] - off[:-1])
    col = col.long()
    total = torch.zeros(n, dtype=torch.float64, device="cuda")
    for root in roots.tolist():
        level = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        paths = torch.zeros(n, dtype=torch.float64, device="cuda")
        level[root], paths[root], d = 0, 1.0, 0
        steps = []
        while True:
            e = level[src] == d
            e &= level[col] == -1
            if not bool(e.any()):
                break
            u, v = src[e], col[e]
            level[v] = d + 1
            paths.index_add_(0, v, paths[u])
            steps.append((u, v))
            d += 1
        delta = torch.zeros(n, dtype=torch.float64, device="cuda")
        for u, v in reversed(steps):
            delta.index_add_(0, u, paths[u] / paths[v] * (1.0 + delta[v]))
        total += delta
    return {"scores": total / total.max(), "levels": None}
