"""The work that users of the engine have it do, as measurable cases.

A case is one call sequence through the public entry points (`PreparedGraph`,
`Session`, `pagerank_multi`, the drop-in `pagerank_csr` and the device-memory
entry `egpr_pagerank_device_noalloc`) on a synthetic graph of stated size:

  solve    one PageRank / personalised PageRank on a prepared graph
  async    the same through enqueue / collect
  device   PageRank on a CSR that the caller holds in device memory
  seeds    a batch of seed-set personalised solves on one graph
  dense    a batch of dense teleport vectors on one graph
  multi    many graphs in one call
  dropin   the drop-in call on a graph not seen before: upload, preparation, solve
  session  a running batched solve that requests join and leave

`graph` is "rmat" (a/b/c/d = 0.57/0.19/0.19/0.05, self-loops and duplicate
pairs removed, vertices >= n dropped) or "er" (uniform pairs, the same rules);
`deg` is the sampled mean out-degree.  tol = 0 runs max_iter sweeps, any other
tol stops on the reference's L1 rule.
"""

import ctypes
import itertools
import math

import numpy as np
import torch

from eggpu_b200 import _native

ALPHA = 0.85
_fresh_id = itertools.count(1)  # ids of graphs that the drop-in call has not seen


def _case(kind, graph, n, deg, weighted=False, tol=1e-6, max_iter=100, name=None, **more):
    c = {"kind": kind, "graph": graph, "n": n, "deg": deg, "weighted": weighted, "tol": tol, "max_iter": max_iter}
    c.update(more)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a request for the smallest graphs of the many-graphs and serving workloads: latency
        _case("solve", "er", 1000, 8, name="solve-er-1k"),
        # the reference's headline small graph, at its own stop rule
        _case("solve", "rmat", 1 << 14, 16, name="solve-rmat14"),
        # a personalised request on a mid-size weighted graph of odd size
        _case("solve", "rmat", 100003, 21, weighted=True, tol=0.0, max_iter=50, pers=True, name="ppr-rmat-100k"),
        # plain PageRank at scale, unweighted: fixed sweeps as the benchmark times them
        _case("solve", "rmat", 1 << 22, 16, tol=0.0, max_iter=20, name="solve-rmat22"),
        # the largest configuration: 529 M weighted edges
        _case("solve", "rmat", 1 << 25, 16, weighted=True, tol=0.0, max_iter=20, name="solve-rmat25w"),
        # a graph without hubs (every gather equally likely), FP32 result, asynchronous entry
        _case("async", "er", 1500007, 11, tol=0.0, max_iter=30, correction=False, name="async-er-1.5m"),
        # a framework that owns device memory, a converging solve with the usual sweep limit
        _case("device", "rmat", 50001, 12, weighted=True, name="device-rmat-50k"),
        # the batched personalised benchmark: 256 seed sets, 20 sweeps
        _case("seeds", "rmat", 1 << 20, 16, tol=0.0, max_iter=20, k=256, max_seeds=64, name="seeds-rmat20-k256"),
        # a queue of personalised requests for one serving graph, ragged batch, stop rule per request
        _case("seeds", "rmat", 60013, 24, weighted=True, k=45, max_seeds=16, name="seeds-rmat-60k-k45"),
        # the many-graphs workload: n log-uniform in [1e3, 2e5], mean degree uniform in [8, 32]
        _case("multi", "er", 200000, 32, count=128, name="multi-er-128"),
        # a program that solves each new graph once: everything from the host arrays to the ranks
        _case("dropin", "rmat", 1 << 20, 16, weighted=True, name="dropin-rmat20w"),
        # long requests joining and leaving a running solve
        _case("session", "rmat", 1 << 17, 16, tol=0.0, max_iter=24, k=96, slots=64, max_seeds=16, name="session-rmat17"),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "async", "device", "seeds", "seeds", "dense", "multi", "dropin", "session"])
    graph = rng.choice(["rmat", "rmat", "er"])
    weighted = rng.random() < 0.5
    deg = rng.randint(8, 32)
    fixed = rng.random() < 0.5
    stop = {"tol": 0.0, "max_iter": rng.randint(2, 40)} if fixed else {"tol": 1e-6, "max_iter": 100}
    if kind == "solve":
        pers = rng.random() < 0.3
        n = _size(rng, 500, 1 << (22 if pers else 24))
        if n > 1 << 21:
            deg, stop = min(deg, 16), {"tol": 0.0, "max_iter": 20}
        return _case(kind, graph, n, deg, weighted, pers=pers, correction=rng.random() < 0.8, **stop)
    if kind == "async":
        return _case(kind, graph, _size(rng, 1000, 4000000), deg, weighted, correction=rng.random() < 0.5, **stop)
    if kind == "device":
        return _case(kind, graph, _size(rng, 500, 262144), deg, weighted, correction=rng.random() < 0.8, **stop)
    if kind == "seeds":
        n = _size(rng, 1000, 1 << 20)
        return _case(kind, graph, n, deg, weighted, k=rng.randint(1, 200 if n > 200000 else 300), max_seeds=64, **stop)
    if kind == "dense":
        return _case(kind, graph, _size(rng, 1000, 200000), deg, weighted, k=rng.randint(2, 40), **stop)
    if kind == "multi":
        return _case(kind, graph, _size(rng, 5000, 200000), 32, weighted, count=rng.randint(3, 120), **stop)
    if kind == "dropin":
        return _case(kind, graph, _size(rng, 1000, 4000000), min(deg, 20), weighted, tol=1e-6, max_iter=100)
    return _case("session", graph, _size(rng, 2000, 200000), deg, weighted, k=rng.randint(6, 120), max_seeds=16,
                 slots=rng.choice([32, 64, 96]), tol=0.0, max_iter=rng.randint(4, 40))


# ---- graphs --------------------------------------------------------------------
def _pairs(graph, n, deg, g):
    """Sorted distinct (source << 32 | destination) keys without self-loops."""
    if graph == "er":
        m = n * deg
        s = torch.randint(0, n, (m,), generator=g, device="cuda", dtype=torch.int32)
        d = torch.randint(0, n, (m,), generator=g, device="cuda", dtype=torch.int32)
    else:
        scale = max(1, (n - 1).bit_length())
        m = deg << scale
        s = torch.zeros(m, dtype=torch.int32, device="cuda")
        d = torch.zeros(m, dtype=torch.int32, device="cuda")
        r = torch.empty(m, device="cuda")
        for _ in range(scale):
            r.uniform_(generator=g)
            s.mul_(2).add_(r >= 0.76)
            d.mul_(2).add_((r >= 0.57) & (r < 0.76)).add_(r >= 0.95)
        del r
    keep = s != d
    if graph == "rmat" and n & (n - 1):
        keep &= (s < n) & (d < n)
    key = (s[keep].long() << 32) | d[keep].long()
    del s, d, keep
    key = key.sort().values
    first = torch.ones(key.numel(), dtype=torch.bool, device="cuda")
    torch.ne(key[1:], key[:-1], out=first[1:])
    return key[first]


def _device_csr(graph, n, deg, weighted, seed):
    """(V int32, E int32, W float64 or None) out-edge CSR on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    key = _pairs(graph, n, deg, g)
    V = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    V[1:] = torch.bincount(key >> 32, minlength=n).cumsum(0)
    E = (key & 0xFFFFFFFF).to(torch.int32)
    W = (1.0 - torch.rand(E.numel(), generator=g, device="cuda")).double() if weighted else None
    return V.to(torch.int32), E, W


def _host(t):
    """A page-locked copy (the caching allocator keeps such memory for the next copy)."""
    if t is None:
        return None
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _graphs(case, seed):
    """(n, deg, seed) of every graph of the case."""
    if case["kind"] != "multi":
        return [(case["n"], case["deg"], seed)]
    rng = np.random.default_rng(case["n"] * 1000 + case["count"])  # the sizes belong to the case
    ns = np.exp(rng.uniform(math.log(1000), math.log(case["n"]), case["count"])).astype(int)
    ds = rng.integers(8, case["deg"] + 1, case["count"])
    return [(int(n), int(d), seed * 1009 + i) for i, (n, d) in enumerate(zip(ns, ds))]


def _seed_sets(case, seed):
    rng = np.random.default_rng(seed)
    sizes = rng.integers(1, case["max_seeds"] + 1, case["k"])
    return [np.unique(rng.integers(0, case["n"], s)).astype(np.int32) for s in sizes]


def _teleports(case, seed):
    """Dense non-negative teleport vectors, a tenth of the entries nonzero."""
    rng = np.random.default_rng(seed)
    k, n = case.get("k", 1), case["n"]
    t = rng.random((k, n)) * (rng.random((k, n)) < 0.1)
    t[:, 0] += 0.5
    return t


# ---- prepare and run -------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    pinned = lambda *shape: _native.pinned_empty(shape)  # noqa: E731
    opts = {"alpha": ALPHA, "max_iter": case["max_iter"], "tol": case["tol"], "correction": case.get("correction", True)}
    s = {"kind": kind, "opts": opts}
    if kind == "multi":
        s["graphs"] = [_native.PreparedGraph(*map(_host, _device_csr(case["graph"], n, d, case["weighted"], sd)))
                       for n, d, sd in _graphs(case, seed)]
        s["out"] = pinned(sum(g.n for g in s["graphs"]))
        ends = np.cumsum([g.n for g in s["graphs"]])
        s["outs"] = [s["out"][e - g.n:e] for g, e in zip(s["graphs"], ends)]
        return s
    V, E, W = _device_csr(case["graph"], case["n"], case["deg"], case["weighted"], seed)
    if kind == "dropin":  # the program's own arrays: ordinary pageable memory
        s["csr"] = (V.cpu().numpy(), E.cpu().numpy(), None if W is None else W.cpu().numpy())
        s["out"] = pinned(case["n"])
        return s
    s["graph"] = pg = _native.PreparedGraph(_host(V), _host(E), _host(W))
    if kind in ("solve", "async"):
        s["out"] = pinned(pg.n)
        s["pers"] = _teleports(case, seed)[0] if case.get("pers") else None
    elif kind == "device":
        row, col, w, _dangling, outw = pg.export_inbound()
        up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        s["nnz"] = int(row[-1])
        s["inputs"] = (up(row), up(col), up(w) if case["weighted"] else None, up(outw))
        s["out"] = torch.empty(pg.n, dtype=torch.float64, device="cuda")
    elif kind == "dense":
        s["teleport"] = _teleports(case, seed)
        s["out"] = pinned(case["k"], pg.n)
    else:
        s["sets"] = _seed_sets(case, seed)
        s["out"] = pinned(case["k"], pg.n)
        s["slots"] = case.get("slots")
    return s


def _run_device(s):
    row, col, w, outw = s["inputs"]
    o = s["opts"]
    ptr = lambda t: ctypes.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731
    stats = _native.EgprStats()
    _native.check(_native.lib.egpr_pagerank_device_noalloc(
        s["graph"].n, s["nnz"], ptr(row), ptr(col), ptr(w), ptr(outw), o["alpha"], o["max_iter"], o["tol"],
        0 if o["correction"] else _native.EGPR_FLAG_NO_CORRECTION, ptr(s["out"]), None, ctypes.byref(stats)))
    return s["out"], stats.iterations


def _run_session(s):
    """Requests arrive 16 at a time between steps, wait for free slots, and
    leave in the order in which they came (they ask for equal sweep counts)."""
    o, sets, out = s["opts"], s["sets"], s["out"]
    sess = _native.Session(s["graph"], alpha=o["alpha"], tol=o["tol"], slots=s["slots"])
    request, nxt, left = {}, 0, len(sets)
    sweeps = np.zeros(len(sets), np.int64)
    try:
        while left:
            room = min(16, sess.info()["free"], len(sets) - nxt)
            if room:
                for j, slot in enumerate(sess.admit(sets[nxt:nxt + room], max_iter=o["max_iter"])):
                    request[slot] = nxt + j
                nxt += room
            done = sorted(sess.step(8), key=request.get)
            if done:
                first = request[done[0]]
                _ranks, stats = sess.collect(done, correction=o["correction"], out=out[first:first + len(done)])
                for slot, st in zip(done, stats):
                    sweeps[request.pop(slot)] = st["iterations"]
                left -= len(done)
    finally:
        sess.close()
    return out, sweeps


def run(s):
    kind, o = s["kind"], s["opts"]
    if kind == "solve":
        ranks, st = s["graph"].pagerank(personalization=s["pers"], out=s["out"], **o)
        return ranks, st["iterations"]
    if kind == "async":
        s["graph"].enqueue(**o)
        ranks, st = s["graph"].collect(out=s["out"])
        return ranks, st["iterations"]
    if kind == "device":
        return _run_device(s)
    if kind == "session":
        return _run_session(s)
    if kind == "dropin":
        ranks, _seconds = _native.pagerank_csr(*s["csr"], next(_fresh_id), o["alpha"], o["max_iter"], o["tol"], out=s["out"])
        return ranks
    if kind == "multi":
        _outs, st = _native.pagerank_multi(s["graphs"], out=s["outs"], **o)
        return s["out"], np.array([t["iterations"] for t in st])
    if kind == "dense":
        ranks, st = s["graph"].pagerank_batch(s["teleport"], out=s["out"], **o)
    else:
        ranks, st = s["graph"].pagerank_seeds(s["sets"], out=s["out"], **o)
    return ranks, np.array([t["iterations"] for t in st])


# ---- what a pass needs, and what it should give ------------------------------------
def work(case):
    """Bytes: per sweep and graph the inbound CSR, once per batch of columns,
    and per column two FP32 rank vectors read and two written; the host
    arrays of a new graph; the FP64 result.  A converging solve is counted
    with the sweeps that such graphs take."""
    total = flops = 0
    for n, deg, _ in _graphs(case, 0):
        m = deg * (n if case["graph"] == "er" else 1 << max(1, (n - 1).bit_length()))
        k = case.get("k", 1) if case["kind"] in ("seeds", "dense", "session") else 1
        sweeps = case["max_iter"] if case["tol"] == 0 else max(1, round(math.log(0.4 / (case["tol"] * n)) / math.log(2.2))) if case["tol"] * n < 0.4 else 1
        sweep = 4 * (n + 1) + m * (8 if case["weighted"] else 4) + k * 16 * n
        total += sweeps * sweep + 8 * n * k
        if case["kind"] == "dropin":
            total += 4 * (n + 1) + m * (12 if case["weighted"] else 4)
        if case["kind"] == "dense" or case.get("pers"):
            total += 8 * n * k
        flops += sweeps * 2 * m * k
    return {"bytes": total, "flops": flops}


def tolerance(case):
    # FP32 sums in another order; the last sweep is FP64 unless it is switched off
    return {"rel": 1e-6, "max": 1e-5}


def _exact_graph(case, n, deg, seed, teleports=None):
    """FP64 ranks (k, n) and sweep counts of one graph by the plain power iteration."""
    V, E, W = _device_csr(case["graph"], n, deg, case["weighted"], seed)
    V = V.long()
    src = torch.repeat_interleave(torch.arange(n, device="cuda"), V[1:] - V[:-1])
    w = W if W is not None else torch.ones(E.numel(), dtype=torch.float64, device="cuda")
    outw = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, src, w)
    order = torch.argsort(E, stable=True)
    row = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    row[1:] = torch.bincount(E, minlength=n).cumsum(0)
    del E, V
    col = src[order]
    val = w[order] / outw[col]
    del src, order, w
    A = torch.sparse_csr_tensor(row.to(torch.int32), col.to(torch.int32), val, (n, n), check_invariants=False)
    dangling = outw <= 1e-15
    P = torch.full((n, 1), 1.0 / n, dtype=torch.float64, device="cuda") if teleports is None else teleports
    k = P.shape[1]
    X = torch.full((n, k), 1.0 / n, dtype=torch.float64, device="cuda")
    count = np.zeros(k, np.int64)
    live = torch.ones(k, dtype=torch.bool, device="cuda")
    for _ in range(case["max_iter"]):
        mass = X[dangling].sum(0)
        Y = (A @ X) * ALPHA + (1.0 - ALPHA) * P + ALPHA * mass / n
        err = (Y - X).abs().sum(0)
        X = torch.where(live, Y, X)
        count += live.cpu().numpy()
        live &= ~(err < case["tol"] * n)
        if not bool(live.any()):
            break
    return (X / X.sum(0)).T.contiguous(), count


def exact(case, seed):
    kind = case["kind"]
    if kind == "multi":
        got = [_exact_graph(case, n, d, sd) for n, d, sd in _graphs(case, seed)]
        return torch.cat([r[0] for r, _ in got]), np.array([c[0] for _, c in got])
    n, P = case["n"], None
    if kind == "dense" or case.get("pers"):
        P = torch.from_numpy(_teleports(case, seed)).cuda().T
        P = P / P.sum(0)
    elif kind in ("seeds", "session"):
        P = torch.zeros(n, case["k"], dtype=torch.float64, device="cuda")
        for j, ids in enumerate(_seed_sets(case, seed)):
            P[torch.from_numpy(ids).long().cuda(), j] = 1.0 / len(ids)
    ranks, count = _exact_graph(case, n, case["deg"], seed, P)
    if kind == "dropin":
        return ranks[0]
    if kind in ("solve", "async", "device"):
        return ranks[0], int(count[0])
    return ranks, count
