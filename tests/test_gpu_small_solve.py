"""The one-kernel solve of small graphs at its edges: rows around the lengths where a
few lanes, a warp and the whole CTA take over, each number of lanes per row, one and
many CTAs, through the prepared graph and through the no-allocation entry.  Compared
with the FP64 oracle; L1 <= 1e-6 is the engine's parity bar."""

import ctypes

import numpy as np
import pytest

from eggpu_b200 import _native
from oracle import oracle

pytestmark = pytest.mark.gpu


def _csr(n, src, dst, weighted):
    order = np.lexsort((dst, src))
    src, dst = src[order], dst[order]
    V = np.zeros(n + 1, np.int32)
    V[1:] = np.cumsum(np.bincount(src, minlength=n))
    W = (1.0 - np.random.default_rng(n).random(len(dst), np.float32)).astype(np.float64) if weighted else None
    return V, dst.astype(np.int32), W


def _graph(n, degree, row, weighted):
    """Random pairs, and one row (n // 2) of `row` entries."""
    rng = np.random.default_rng(n + row)
    src = np.concatenate([rng.integers(0, n, n * degree), np.arange(row) % n])
    dst = np.concatenate([rng.integers(0, n, n * degree), np.full(row, n // 2)])
    return _csr(n, src, dst, weighted)


def _noalloc(pg, weighted, **o):
    import torch

    row, col, w, _dangling, outw = pg.export_inbound()
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (row, col, w, outw)]
    out = torch.full((pg.n,), float("nan"), dtype=torch.float64, device="cuda")
    st = _native.EgprStats()
    p = [ctypes.c_void_p(t.data_ptr()) for t in dev]
    _native.check(_native.lib.egpr_pagerank_device_noalloc(
        pg.n, int(row[-1]), p[0], p[1], p[2] if weighted else None, p[3], 0.85, o["max_iter"], o["tol"],
        0 if o["correction"] else 1, ctypes.c_void_p(out.data_ptr()), None, ctypes.byref(st)))
    return out.cpu().numpy(), st.as_dict()


@pytest.mark.parametrize("correction", [True, False])
@pytest.mark.parametrize("n,degree,row,weighted", [
    (1, 1, 1, False), (3, 2, 0, True), (33, 3, 127, True), (1000, 3, 128, False), (1000, 8, 129, True),
    (2049, 10, 1023, True), (2049, 10, 1024, False), (2050, 30, 1025, True), (4096, 30, 9000, True),
    (16384, 12, 20000, False), (20011, 5, 3000, True),
    # more than 96 entries per row: a warp per row; rows around four times the mean, from
    # which the whole CTA takes over; and few rows, of which the CTA takes all above 1024
    (40, 99, 0, False), (700, 400, 1200, True), (700, 400, 1201, False), (700, 400, 1900, True),
    (5, 3000, 0, True), (9, 1024, 0, False)])
def test_small_solve_at_row_length_edges(monkeypatch, n, degree, row, weighted, correction):
    monkeypatch.delenv("EGPR_SMALL_NNZ", raising=False)
    V, E, W = _graph(n, degree, row, weighted)
    pg = _native.PreparedGraph(V, E, W)
    o = {"max_iter": 7, "tol": 0.0, "correction": correction}
    ref, _, _ = oracle.pagerank_pull(V, E, W, alpha=0.85, max_iter=7, tol=0.0)
    for got, st in (pg.pagerank(**o), _noalloc(pg, weighted, **o)):
        assert st["iterations"] == 7 and st["converged"] == 0
        assert np.abs(got - ref).sum() <= 1e-6
    again, _ = pg.pagerank(**o)
    assert np.array_equal(again, pg.pagerank(**o)[0])  # the same bits every time
    p = np.zeros(n)
    p[[0, n - 1]] = (1.0, 3.0)
    got, _ = pg.pagerank(personalization=p, **o)
    ref, _, _ = oracle.pagerank_pull(V, E, W, alpha=0.85, max_iter=7, tol=0.0, teleport=p / p.sum())
    assert np.abs(got - ref).sum() <= 1e-6
    rule, st = pg.pagerank(max_iter=100, tol=1e-7)
    ref, it, _ = oracle.pagerank_pull(V, E, W, alpha=0.85, max_iter=100, tol=1e-7)
    if 1e-7 * n > 1e-6:  # the stop rule is above FP32 resolution
        assert abs(st["iterations"] - it) <= 1 and st["converged"] == 1
    assert np.abs(rule - ref).sum() <= max(1e-6, 1e-7 * n)
    pg.close()


def test_solves_beside_others_give_the_same_bits(monkeypatch):
    """A solve beside others takes fewer CTAs; its sums do not depend on their number."""
    import threading

    monkeypatch.delenv("EGPR_SMALL_NNZ", raising=False)
    graphs = [_native.PreparedGraph(*_graph(n, d, row, w)) for n, d, row, w in
              [(16384, 12, 3000, False), (9000, 20, 500, True), (1000, 8, 0, False), (2000, 90, 2500, True)] * 3]
    o = {"max_iter": 30, "tol": 0.0}
    alone = [pg.pagerank(**o)[0].copy() for pg in graphs]
    wrong = []

    def solve(i):
        for _ in range(20):
            if not np.array_equal(graphs[i].pagerank(**o)[0], alone[i]):
                wrong.append(i)

    threads = [threading.Thread(target=solve, args=(i,)) for i in range(len(graphs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    for pg in graphs:  # all enqueued, then collected
        pg.enqueue(**o)
    for pg, want in zip(graphs, alone):
        assert np.array_equal(pg.collect()[0], want)
        pg.close()


def test_noalloc_solve_can_be_captured():
    """The work is only enqueued (stats NULL), so a stream capture takes it; a replay
    solves again."""
    import torch

    V, E, W = _graph(3000, 9, 700, True)
    pg = _native.PreparedGraph(V, E, W)
    want, _ = _noalloc(pg, True, max_iter=9, tol=0.0, correction=True)
    row, col, w, _dangling, outw = pg.export_inbound()
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (row, col, w, outw)]
    out = torch.zeros(pg.n, dtype=torch.float64, device="cuda")
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        _native.check(_native.lib.egpr_pagerank_device_noalloc(
            pg.n, int(row[-1]), *[ctypes.c_void_p(t.data_ptr()) for t in dev], 0.85, 9, 0.0, 0,
            ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), None))
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), want)
