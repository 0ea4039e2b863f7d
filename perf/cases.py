"""The calls whose speed this repository is held to, over the ranges they are used in.

Graphs are undirected unless a case says otherwise and are built on the device from seeded R-MAT pairs
(a, b, c, d = 0.57, 0.19, 0.19, 0.05, edge factor 16 as in the benchmark) or from uniform-random pairs.
Results stay in device memory: where a method of GraphVine returns host arrays only, the call behind it in
the C ABI (include/gv.h) is made with device pointers, as a C++ program makes it.

Kinds of case:
  stream     a sliding window over an edge stream: insert the new batch, delete the expired one, compact,
             read the adjacency as CSR and the degrees; then the same step back, so that a pass can be repeated
  window     a window of many uneven update batches in one batch_run, replayed from its CUDA graph, then its
             inverse; the adjacency is read after the first
  pagerank   static_pagerank with its default arguments
  ppr        a batch of personalised PageRank queries
  triangles  the exact triangle count, total only or with the count each vertex owns
  bc         betweenness centrality from a set of sources
  gradient   weighted PageRank on a directed store and its gradient by every edge weight
  ingest     Matrix-Market text in device memory to edge arrays
"""
import ctypes
import math

import numpy as np
import torch

import gv_b200
from gv_b200 import _lib

DEV = "cuda:0"
ALPHA, EPS, MAX_ITER = 0.85, 1e-6, 100   # static_pagerank's and ppr_batch's defaults
TOL, TOL_ITER = 1e-7, 200                # wpr_forward's and wpr_backward's defaults
MEM = _lib.GV_MEM_DEVICE


def listed():
    return [
        # a service's smallest update: 1,000 edges in and 1,000 out of a small resident graph
        {"name": "stream_small", "kind": "stream", "graph": "rmat", "n": 1 << 14, "pairs": 16 << 14, "batch": 1000,
         "block": 32, "tpv": 8},
        # the benchmark's step: 1M updates, half inserts and half deletes, on the scale-22 graph
        {"name": "stream_large", "kind": "stream", "graph": "rmat", "n": 1 << 22, "pairs": 16 << 22, "batch": 500_000,
         "block": 128, "tpv": 16},
        # the benchmark's batching workload at a smaller scale: 64 uneven batches, Zipf-skewed sources
        {"name": "window", "kind": "window", "graph": "rmat", "n": 1 << 20, "pairs": 16 << 20, "batches": 64,
         "smallest": 1000, "largest": 200_000, "block": 128, "tpv": 8},
        # PageRank of a graph that a user tries things out on: launches and latency count
        {"name": "pagerank_small", "kind": "pagerank", "graph": "rmat", "n": 1 << 14, "pairs": 16 << 14, "block": 128,
         "tpv": 8},
        # PageRank of the benchmark's step: ten batches of uniform-random inserts later, which link vertices that
        # R-MAT leaves alone and make it take more sweeps
        {"name": "pagerank_large", "kind": "pagerank", "graph": "rmat", "n": 1 << 22, "pairs": 16 << 22,
         "added": 5_000_000, "block": 128, "tpv": 16},
        # 32 queries at once, the most that one call takes
        {"name": "ppr_batch", "kind": "ppr", "graph": "rmat", "n": 1 << 20, "pairs": 16 << 20, "queries": 32,
         "block": 128, "tpv": 8},
        # the count per vertex on a mid-sized graph without hubs, of a size that no tile divides
        {"name": "triangles_owner", "kind": "triangles", "graph": "uniform", "n": 100_003, "pairs": 1_600_061,
         "owner": True, "block": 64, "tpv": 8},
        # the total of the benchmark's step
        {"name": "triangles_large", "kind": "triangles", "graph": "rmat", "n": 1 << 22, "pairs": 16 << 22,
         "owner": False, "block": 128, "tpv": 16},
        # one served betweenness request on a small graph: BFS levels are launches
        {"name": "bc_small", "kind": "bc", "graph": "rmat", "n": 1 << 14, "pairs": 16 << 14, "sources": 32,
         "block": 128, "tpv": 8},
        # betweenness from 64 sampled sources
        {"name": "bc_large", "kind": "bc", "graph": "rmat", "n": 1 << 20, "pairs": 16 << 20, "sources": 64,
         "block": 128, "tpv": 8},
        # the benchmark's differentiation workload: forward, adjoint and gradient
        {"name": "gradient", "kind": "gradient", "graph": "rmat", "n": 1 << 20, "pairs": 16 << 20, "block": 128,
         "tpv": 8},
        # a weighted edge list of some 80 MB
        {"name": "ingest", "kind": "ingest", "graph": "rmat", "n": 1 << 18, "pairs": 16 << 18, "values": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["stream", "window", "pagerank", "ppr", "triangles", "bc", "gradient", "ingest"])
    top = {"stream": 1 << 22, "pagerank": 1 << 22, "triangles": 1 << 21, "ingest": 1 << 19}.get(kind, 1 << 20)
    n = _log(rng, 1 << 14, top)
    if rng.random() < 0.25:
        n = 1 << max(14, min(22, n.bit_length() - 1))
    pairs = int(n * rng.uniform(4, 16))
    c = {"kind": kind, "graph": rng.choice(["rmat", "rmat", "uniform"]), "n": n, "pairs": pairs}
    if kind != "ingest":
        c["block"] = rng.choice([32, 64, 128])
        c["tpv"] = rng.choice([4, 8, 16, 32])
    if kind == "stream":
        c["batch"] = _log(rng, 1000, max(1100, min(500_000, pairs // 8)))
    elif kind == "window":
        c["batches"] = rng.randint(4, 64)
        c["smallest"] = 1000
        c["largest"] = _log(rng, 2000, max(2100, min(200_000, pairs // 16)))
    elif kind == "pagerank":
        c["added"] = rng.choice([0, pairs // 13])
    elif kind == "ppr":
        c["queries"] = rng.randint(2, 32)
    elif kind == "triangles":
        c["owner"] = rng.random() < 0.5
    elif kind == "bc":
        c["sources"] = rng.randint(1, 64)
    elif kind == "ingest":
        c["values"] = rng.random() < 0.5
    return c


# ------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _pairs(case, gen):
    """(u, v) int64: the case's raw pairs, self-loops and duplicates among them."""
    n, k = case["n"], case["pairs"]
    if case["graph"] == "uniform":
        return (torch.randint(0, n, (k,), generator=gen, device=DEV),
                torch.randint(0, n, (k,), generator=gen, device=DEV))
    u = torch.zeros(k, dtype=torch.int32, device=DEV)
    v = torch.zeros(k, dtype=torch.int32, device=DEV)
    for _ in range((n - 1).bit_length()):
        r = torch.rand(k, generator=gen, device=DEV)
        u.mul_(2).add_(r >= 0.76)
        v.mul_(2).add_(((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    return u.long() % n, v.long() % n


def _keys(u, v, n, directed=False):
    """Sorted distinct keys of the pairs without self-loops: lo * n + hi, or u * n + v of directed ones."""
    keep = u != v
    u, v = u[keep], v[keep]
    return torch.unique(u * n + v if directed else torch.minimum(u, v) * n + torch.maximum(u, v))


def _fresh(case, count, old, gen, zipf):
    """`count` distinct new edges (keys) in random order that `old` does not hold; Zipf(1.1) or uniform sources."""
    n = case["n"]
    got = torch.empty(0, dtype=torch.int64, device=DEV)
    while got.numel() < count:
        k = 2 * (count - got.numel()) + 64
        if zipf:
            r = torch.rand(k, generator=gen, device=DEV, dtype=torch.float64)
            u = (1.0 - r * (1.0 - n ** -0.1)).pow(-10.0).long().clamp_(1, n) - 1
            u = (u * 0x9E3779B1 + 12345) % n
        else:
            u = torch.randint(0, n, (k,), generator=gen, device=DEV)
        new = _keys(u, torch.randint(0, n, (k,), generator=gen, device=DEV), n)
        at = torch.searchsorted(old, new).clamp_(max=max(old.numel() - 1, 0))
        got = torch.unique(torch.cat([got, new[old[at] != new]]))
        got = got[torch.randperm(got.numel(), generator=gen, device=DEV)[:count]]
    return got


def _split(keys, n, gen=None):
    """int32 endpoints of the keys; with `gen`, each pair in a random order."""
    u, v = (keys // n).int(), (keys % n).int()
    if gen is None:
        return u, v
    flip = torch.rand(u.numel(), generator=gen, device=DEV) < 0.5
    return torch.where(flip, v, u), torch.where(flip, u, v)


def _store(case, entries, spare=0, **more):
    """An empty store that has room for `entries` directed entries and `spare` more."""
    b = case["block"]
    return gv_b200.GraphVine(case["n"], block_size=b, threads_per_vertex=case["tpv"],
                             pool_blocks=case["n"] + (entries + spare) // b + min(case["n"], spare) + spare // b + 1024,
                             **more)


def _insert(g, keys, n, gen):
    """The graph's edges as the user's program loads them: one batch, in no order."""
    order = torch.randperm(keys.numel(), generator=gen, device=DEV)
    g.batch_insert(*_split(keys[order], n, gen))
    g.synchronize()


def _simple_graph(case, seed):
    gen = _gen(seed)
    n = case["n"]
    u, v = _pairs(case, gen)
    if k := case.get("added"):
        more = torch.randint(0, n, (2, k), generator=gen, device=DEV)
        u, v = torch.cat([u, more[0]]), torch.cat([v, more[1]])
    return gen, n, _keys(u, v, n)


def _spans(case):
    """Per batch of a window (inserts, deletes): sizes log-uniform, the insert share uniform in [0.2, 0.8]."""
    r = np.random.default_rng(case["batches"] * case["largest"])
    size = np.exp(r.uniform(math.log(case["smallest"]), math.log(case["largest"]), case["batches"])).astype(np.int64)
    ins = (size * r.uniform(0.2, 0.8, case["batches"])).astype(np.int64)
    return [(int(a), int(b)) for a, b in zip(ins, size - ins)]


def _layout(spans, ins, dele, n, gen):
    """(descs, src, dst) of a window that inserts `ins` and deletes `dele`, batch by batch."""
    parts, descs, i, j, off = [], [], 0, 0, 0
    for a, b in spans:
        parts += [ins[i:i + a], dele[j:j + b]]
        descs.append((off, a, b))
        i, j, off = i + a, j + b, off + a + b
    return (descs, *_split(torch.cat(parts), n, gen))


def _digits(ids, most):
    nd = torch.ones_like(ids)
    for j in range(1, most):
        nd += ids >= 10 ** j
    return nd


def _mtx_entries(case, seed):
    gen = _gen(seed)
    u, v = _pairs(case, gen)
    w = torch.randint(1, 10_000, (u.numel(),), generator=gen, device=DEV) if case["values"] else None
    return u, v, w


def prepare(case, seed):
    kind = case["kind"]
    st = _prepare(kind, case, seed)
    torch.cuda.empty_cache()  # the graph store allocates beside torch
    return st


def _prepare(kind, case, seed):
    if kind == "ingest":
        u, v, w = _mtx_entries(case, seed)
        n, k, most = case["n"], u.numel(), len(str(case["n"]))
        u, v = u + 1, v + 1
        nu, nv = _digits(u, most), _digits(v, most)
        tail = 8 if w is not None else 1           # " 0.dddd\n" or "\n"
        end = torch.cumsum(nu + 1 + nv + tail, 0)
        start = end - (nu + 1 + nv + tail)
        text = torch.full((int(end[-1]),), ord(" "), dtype=torch.uint8, device=DEV)
        for ids, nd, at in ((u, nu, start), (v, nv, start + nu + 1)):
            for j in range(most):
                has = nd > j
                text[(at + nd - 1 - j)[has]] = ((ids // 10 ** j) % 10 + 48)[has].to(torch.uint8)
        text[end - 1] = ord("\n")
        if w is not None:
            text[end - 7] = ord("0")
            text[end - 6] = ord(".")
            for j in range(4):
                text[end - 2 - j] = ((w // 10 ** j) % 10 + 48).to(torch.uint8)
        field = "real" if w is not None else "pattern"
        head = f"%%MatrixMarket matrix coordinate {field} general\n% seeded\n{n} {n} {k}\n".encode()
        return {"case": case, "text": torch.cat([torch.tensor(list(head), dtype=torch.uint8, device=DEV), text])}
    if kind == "gradient":
        gen = _gen(seed)
        n = case["n"]
        keys = _keys(*_pairs(case, gen), n, directed=True)
        u, v = keys // n, (keys % n).int()
        w = 1.0 - 0.9 * torch.rand(keys.numel(), generator=gen, device=DEV)
        off = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
        off[1:] = torch.cumsum(torch.bincount(u, minlength=n), 0)
        c = torch.randn(n, generator=gen, device=DEV)
        g = _store(case, keys.numel(), directed=True, weighted=True)
        g.bulk_build(off, v, w)
        g.synchronize()
        x, lam, grad = (torch.zeros(k, device=DEV) for k in (n, n, case["pairs"]))  # grad: one per entry, the rest 0
        return {"case": case, "g": g, "c": c, "x": x, "lam": lam, "grad": grad}
    gen, n, keys = _simple_graph(case, seed)
    if kind in ("stream", "window"):
        spans = _spans(case) if kind == "window" else [(case["batch"], case["batch"])]
        na, nb = sum(a for a, _ in spans), sum(b for _, b in spans)
        new = _fresh(case, na + nb, keys, gen, kind == "window")
        a, b = new[:na], new[na:]
        # room for both batches at once
        g = _store(case, 2 * (keys.numel() + na + nb), 2 * (na + nb), max_batch_pairs=max(1 << 16, na + nb))
        _insert(g, keys, n, gen)
        g.batch_insert(*_split(b, n))  # the edges that expire are the youngest of their lists
        g.synchronize()
        st = {"case": case, "g": g, "off": torch.empty(n + 1, dtype=torch.int64, device=DEV),
              "dst": torch.full((2 * (case["pairs"] + na),), -1, dtype=torch.int32, device=DEV),
              "deg": torch.empty(n, dtype=torch.int32, device=DEV)}
        if kind == "stream":
            st["a"], st["b"] = _split(a, n, gen), _split(b, n, gen)
        else:
            st["there"] = _layout(spans, a, b, n, gen)
            st["back"] = _layout([(y, x) for x, y in spans], b, a, n, gen)
        return st
    g = _store(case, 2 * keys.numel())
    _insert(g, keys, n, gen)
    st = {"case": case, "g": g}
    if kind == "pagerank":
        st["x"] = torch.empty(n, dtype=torch.float32, device=DEV)
    elif kind == "ppr":
        st["sources"] = _sources(case, seed, case["queries"])
        st["x"] = torch.empty(n, case["queries"], dtype=torch.float32, device=DEV)
    elif kind == "triangles":
        st["owner"] = torch.empty(n, dtype=torch.int64, device=DEV) if case["owner"] else None
    elif kind == "bc":
        st["sources"] = torch.from_numpy(_sources(case, seed, case["sources"]).view(np.int32)).to(DEV)
        st["bc"] = torch.empty(n, dtype=torch.float32, device=DEV)
    return st


def _sources(case, seed, k):
    return np.random.default_rng(seed + 7).choice(case["n"], size=k, replace=False).astype(np.uint32)


# --------------------------------------------------------------------- calls
def _ok(status):
    if status:
        raise RuntimeError(f"status {status}: {_lib.lib().gv_last_error_string().decode(errors='replace')}")


def _adjacency(st):
    """The adjacency in the program's own buffers, which hold any graph of this case (the rest of dst stays -1)."""
    _ok(_lib.lib().gv_export_csr(st["g"]._h, st["off"].data_ptr(), st["dst"].data_ptr(), None, st["dst"].numel(), MEM,
                                 None))
    return st["off"], st["dst"]


def run(st):
    case, g, L = st["case"], st.get("g"), _lib.lib()
    kind = case["kind"]
    if kind == "stream":
        g.batch_insert(*st["a"])
        g.batch_delete(*st["b"])
        g.compaction()
        off, dst = _adjacency(st)
        g.batch_insert(*st["b"])
        g.batch_delete(*st["a"])
        g.compaction()
        _ok(L.gv_degrees(g._h, st["deg"].data_ptr(), MEM, None))
        return {"offsets": off, "dst": dst, "degrees": st["deg"]}
    if kind == "window":
        g.batch_run(st["there"], compact=True, graph=True)
        off, dst = _adjacency(st)
        g.batch_run(st["back"], compact=True, graph=True)
        _ok(L.gv_degrees(g._h, st["deg"].data_ptr(), MEM, None))
        return {"offsets": off, "dst": dst, "degrees": st["deg"]}
    if kind == "pagerank":
        # the number of sweeps, which hangs on the last bits of the residual, is not handed on
        return g.static_pagerank(ALPHA, EPS, MAX_ITER, out=st["x"])[0]
    if kind == "ppr":
        return g.ppr_batch(st["sources"], ALPHA, EPS, MAX_ITER, out=st["x"])[0]
    if kind == "triangles":
        total = ctypes.c_uint64()
        own = st["owner"]
        _ok(L.gv_tc(g._h, None if own is None else own.data_ptr(), ctypes.byref(total), MEM, None))
        return {"total": total.value} if own is None else {"total": total.value, "owner": own}
    if kind == "bc":
        _ok(L.gv_bc(g._h, st["sources"].data_ptr(), case["sources"], st["bc"].data_ptr(), MEM, None))
        return st["bc"]
    if kind == "gradient":
        sw = ctypes.c_int32()
        _ok(L.gv_wpr_forward(g._h, ALPHA, TOL, TOL_ITER, st["x"].data_ptr(), ctypes.byref(sw), MEM, None))
        _ok(L.gv_wpr_backward(g._h, ALPHA, TOL, TOL_ITER, st["x"].data_ptr(), st["c"].data_ptr(), 0, st["grad"].data_ptr(),
                              st["grad"].numel(), st["lam"].data_ptr(), ctypes.byref(sw), MEM, None))
        return {"x": st["x"], "lambda": st["lam"], "grad": st["grad"]}
    _, src, dst, val = gv_b200.mtx_parse(st["text"], with_values=case["values"])
    return {"src": src, "dst": dst, "val": val} if case["values"] else {"src": src, "dst": dst}


def work(case):
    """What a pass cannot do without.  Edges kept of the raw pairs: about 0.95 of them on the large graphs."""
    n, m = case["n"], 2 * 0.95 * case["pairs"]
    kind = case["kind"]
    if kind == "stream":  # both steps: the pairs in, an entry written or taken out in both lists; the CSR out
        return {"bytes": 4 * case["batch"] * (8 + 8 + 8) + 2 * 4 * m + 8 * n + 2 * 4 * n, "flops": 0}
    if kind == "window":
        total = sum(a + b for a, b in _spans(case))
        return {"bytes": 2 * total * (8 + 8 + 8) + 2 * 4 * m + 8 * n + 2 * 4 * n, "flops": 0}
    if kind == "pagerank":  # some 10 sweeps, 15 on R-MAT, 39 with added edges: each over the adjacency and three vectors
        sweeps = 10 if case["graph"] == "uniform" else 39 if case.get("added") else 15
        return {"bytes": sweeps * (4 * m + 12 * n), "flops": sweeps * 2 * m}
    if kind == "ppr":
        k = case["queries"]
        return {"bytes": 16 * (4 * m + 12 * k * n), "flops": 16 * 2 * m * k}
    if kind == "triangles":
        return {"bytes": 4 * m + (8 * n if case["owner"] else 8), "flops": 0}
    if kind == "bc":  # each of some 7 levels of both halves once over the adjacency, per source sigma, delta and level
        return {"bytes": 2 * 4 * m + case["sources"] * 32 * n, "flops": 2 * 2 * m * case["sources"]}
    if kind == "gradient":  # about 63 and 114 sweeps over entries and weights, then one gradient each
        m /= 2
        return {"bytes": 177 * (8 * m + 12 * n) + 8 * m, "flops": 177 * 2 * m}
    k, d = case["pairs"], len(str(n))
    line = 2 * d + 1 + (8 if case["values"] else 1)
    return {"bytes": k * (line + 8 + (4 if case["values"] else 0)), "flops": 0}


# --------------------------------------------------------------------- exact
def _csr(rows, cols, vals, n):
    order = torch.argsort(rows * n + cols)
    crow = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    crow[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    return torch.sparse_csr_tensor(crow, cols[order], vals[order], (n, n))


def _adj64(case, seed):
    """The undirected graph as a 0/1 matrix in 64 bits, and its degrees."""
    _, n, keys = _simple_graph(case, seed)
    u, v = keys // n, keys % n
    rows, cols = torch.cat([u, v]), torch.cat([v, u])
    deg = torch.bincount(rows, minlength=n).double()
    return n, _csr(rows, cols, torch.ones(rows.numel(), dtype=torch.float64, device=DEV), n), deg


def _power(step, x, tol, most):
    """x <- step(x) until every column's L1 step is under tol."""
    for _ in range(most):
        y = step(x)
        d = (y - x).abs().sum(0)
        x = y
        if bool((d < tol).all()):
            break
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "pagerank":
        n, adj, deg = _adj64(case, seed)
        inv = torch.where(deg > 0, 1.0 / deg, 0.0)[:, None]
        x = torch.full((n, 1), 1.0 / n, dtype=torch.float64, device=DEV)
        return _power(lambda x: (1 - ALPHA) / n + ALPHA * (adj @ (x * inv)), x, EPS, MAX_ITER)[:, 0]
    if kind == "ppr":
        n, adj, deg = _adj64(case, seed)
        inv = torch.where(deg > 0, 1.0 / deg, 0.0)[:, None]
        k = case["queries"]
        src = torch.from_numpy(_sources(case, seed, k).astype(np.int64)).to(DEV)
        e = torch.zeros(n, k, dtype=torch.float64, device=DEV)
        e[src, torch.arange(k, device=DEV)] = 1.0
        return _power(lambda x: (1 - ALPHA) * e + ALPHA * (adj @ (x * inv)), e, EPS, MAX_ITER)
    if kind == "bc":
        n, adj, _ = _adj64(case, seed)
        k = case["sources"]
        src = torch.from_numpy(_sources(case, seed, k).astype(np.int64)).to(DEV)
        at = torch.arange(k, device=DEV)
        dist = torch.full((n, k), -1, dtype=torch.int16, device=DEV)
        sigma = torch.zeros(n, k, dtype=torch.float64, device=DEV)
        dist[src, at], sigma[src, at] = 0, 1.0
        level = 0
        while True:
            y = adj @ (sigma * (dist == level))
            new = (dist < 0) & (y > 0)
            if not bool(new.any()):
                break
            level += 1
            dist[new] = level
            sigma += y * new
        delta = torch.zeros_like(sigma)
        for lv in range(level, 0, -1):
            on = dist == lv
            y = adj @ torch.where(on, (1.0 + delta) / sigma.clamp(min=1.0), 0.0)
            delta += torch.where(dist == lv - 1, sigma * y, 0.0)
        delta[src, at] = 0.0
        return delta.sum(1)
    if kind == "gradient":
        gen = _gen(seed)
        n = case["n"]
        keys = _keys(*_pairs(case, gen), n, directed=True)
        w = (1.0 - 0.9 * torch.rand(keys.numel(), generator=gen, device=DEV)).double()
        c = torch.randn(n, generator=gen, device=DEV).double()
        u, v = keys // n, keys % n
        s = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, u, w)
        p = w / s[u]
        fwd, back = _csr(v, u, p, n), _csr(u, v, p, n)
        x = torch.full((n, 1), 1.0 / n, dtype=torch.float64, device=DEV)
        x = _power(lambda x: (1 - ALPHA) / n + ALPHA * (fwd @ x), x, TOL, TOL_ITER)[:, 0]
        lam = _power(lambda y: c[:, None] + ALPHA * (back @ y), c[:, None], TOL, TOL_ITER)[:, 0]
        grad = torch.zeros(case["pairs"], dtype=torch.float64, device=DEV)
        grad[:keys.numel()] = x[u] * (ALPHA * lam[v] - lam[u] + c[u]) / s[u]
        return {"x": x, "lambda": lam, "grad": grad}
    if kind == "ingest" and case["values"]:
        return {"src": None, "dst": None, "val": _mtx_entries(case, seed)[2].double() / 10_000}
    return None  # whole numbers
