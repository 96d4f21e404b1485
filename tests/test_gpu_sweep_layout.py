"""The blocked layout of the single-vector sweep at the sizes where it can go
wrong: sources around a block's size, runs around a tile's and a chunk's, rows around
a row tile's, one row or one source with every entry, and the layout without blocks.
Ranks are compared with the FP64 oracle; L1 <= 1e-6 is the engine's parity bar (FP32
iterates of ranks that sum to 1, the last sweep in FP64)."""

import numpy as np
import pytest

from eggpu_b200 import _native
from oracle import oracle

pytestmark = pytest.mark.gpu

BLOCK = 22528  # sources per block


def _csr(n, src, dst, weighted, seed):
    order = np.lexsort((dst, src))
    src, dst = src[order], dst[order]
    V = np.zeros(n + 1, np.int32)
    V[1:] = np.cumsum(np.bincount(src, minlength=n))
    W = (1.0 - np.random.default_rng(seed).random(len(dst), np.float32)).astype(np.float64) if weighted else None
    return V, dst.astype(np.int32), W


def _ring(n):
    """Every vertex has one out-edge: n sources."""
    u = np.arange(n)
    return u, (u + 1) % n


def _check(V, E, W, sweeps=6):
    pg = _native.PreparedGraph(V, E, W)
    try:
        for correction in (True, False):
            got, st = pg.pagerank(alpha=0.85, max_iter=sweeps, tol=0.0, correction=correction)
            ref, _, _ = oracle.pagerank_pull(V, E, W, alpha=0.85, max_iter=sweeps, tol=0.0)
            assert st["iterations"] == sweeps
            assert np.abs(got - ref).sum() <= 1e-6
            again, _ = pg.pagerank(alpha=0.85, max_iter=sweeps, tol=0.0, correction=correction)
            assert np.array_equal(got, again)  # order-free sums: the same bits every time
        p = np.zeros(len(V) - 1)
        p[[0, len(p) // 2, len(p) - 1]] = (1.0, 2.0, 3.0)
        got, _ = pg.pagerank(alpha=0.85, max_iter=sweeps, tol=0.0, personalization=p)
        ref, _, _ = oracle.pagerank_pull(V, E, W, alpha=0.85, max_iter=sweeps, tol=0.0, teleport=p / p.sum())
        assert np.abs(got - ref).sum() <= 1e-6
    finally:
        pg.close()


@pytest.fixture(params=["blocks", "one block"])
def layout(request, monkeypatch):
    monkeypatch.setenv("EGPR_SMALL_NNZ", "0")  # small graphs too take the sweep's path
    if request.param == "one block":
        monkeypatch.setenv("EGPR_MAX_CELLS", "1")


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("n", [BLOCK - 1, BLOCK, BLOCK + 1, 2 * BLOCK + 33])
def test_sources_around_a_block(layout, n, weighted):
    u, v = _ring(n)
    rng = np.random.default_rng(n)
    extra = rng.integers(0, n, (2, 40000))
    extra[1, :20000] = rng.integers(0, 40, 20000)  # rows with runs in every block
    V, E, W = _csr(n, np.concatenate([u, extra[0]]), np.concatenate([v, extra[1]]), weighted, n)
    _check(V, E, W)


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("m", [1, 31, 255, 256, 257, 1024, 1025, 5000])
def test_one_row_with_every_entry(layout, m, weighted):
    n = m + 7
    V, E, W = _csr(n, np.arange(1, m + 1), np.zeros(m, int), weighted, m)
    _check(V, E, W)


@pytest.mark.parametrize("n", [31, 32, 33, 255, 257, 12289, 50001])
def test_one_source_with_every_entry_and_empty_rows(layout, n):
    d = np.arange(1, n, 2)
    V, E, W = _csr(n, np.zeros(len(d), int), d, True, n)
    _check(V, E, W)


CHUNKED = 2 * 32 * 1024  # entries per SM from which chunks have four tiles: two of them for each of 32 warps


def _long_runs(n, m, seed, weighted):
    """A few rows hold most of a block's entries."""
    rng = np.random.default_rng(seed)
    src = np.concatenate([np.arange(n), rng.integers(0, n, m)])
    dst = np.concatenate([(np.arange(n) + 1) % n, np.where(rng.random(m) < 0.7, rng.integers(0, 5, m), rng.integers(0, n, m))])
    return _csr(n, src, dst, weighted, seed + 1)


def test_long_runs_cross_chunks():
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    V, E, W = _long_runs(30011, CHUNKED * sms, 5, True)
    assert len(E) >= CHUNKED * sms
    _check(V, E, W, sweeps=3)


def test_every_cut_of_a_chunked_plan_gives_the_same_bits():
    """Row sums are order-free and runs end at fixed chunks, so the cuts between the CTAs
    of the first phase change nothing; one graph per solve and two in one plan."""
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    graphs = [_native.PreparedGraph(*_long_runs(n, CHUNKED * sms + n, n, False)) for n in (70001, 30011)]
    o = {"max_iter": 3, "tol": 0.0}
    first = [pg.pagerank(**o)[0] for pg in graphs]
    for row_cost in (0, 1, 2, 3, 5, 7, 8, 13, 33, 64):
        for pg, want in zip(graphs, first):
            pg.set_tuning(row_cost=row_cost)
            assert np.array_equal(pg.pagerank(**o)[0], want), row_cost
        outs, _ = _native.pagerank_multi(graphs, **o)
        assert all(np.array_equal(a, b) for a, b in zip(outs, first)), row_cost
    for pg in graphs:
        pg.close()


@pytest.mark.parametrize("row_tiles", [1, 3, 64])
def test_any_tuning_gives_the_same_ranks(layout, row_tiles):
    """Row tiles of all sizes: other cuts of the rows change the order of no sum."""
    rng = np.random.default_rng(8)
    n = 60013
    V, E, W = _csr(n, rng.integers(0, n, 700000), np.minimum(rng.zipf(1.3, 700000) - 1, n - 1), True, 9)
    pg = _native.PreparedGraph(V, E, W)
    o = {"max_iter": 5, "tol": 0.0}
    ref, _, _ = oracle.pagerank_pull(V, E, W, alpha=0.85, **o)
    pg.set_tuning(chunks_per_warp=row_tiles, row_cost=0 if row_tiles == 1 else row_tiles)
    got, _ = pg.pagerank(**o)
    assert np.abs(got - ref).sum() <= 1e-6
    assert np.array_equal(got, pg.pagerank(**o)[0])
    pg.close()


@pytest.mark.parametrize("tol,max_iter", [(0.0, 7), (1e-9, 200)])
def test_sweep_on_a_callers_stream(layout, tol, max_iter):
    import torch

    rng = np.random.default_rng(12)
    n = 30011
    V, E, W = _csr(n, rng.integers(0, n, 300000), rng.integers(0, n, 300000), True, 13)
    pg = _native.PreparedGraph(V, E, W)
    o = {"max_iter": max_iter, "tol": tol}
    want, st = pg.pagerank(**o)
    ref, it, _ = oracle.pagerank_pull(V, E, W, alpha=0.85, **o)
    assert np.abs(want - ref).sum() <= 1e-6 and abs(st["iterations"] - it) <= 1
    stream = torch.cuda.Stream()
    pg.set_stream(stream.cuda_stream)
    busy = torch.zeros(1 << 24, device="cuda")
    with torch.cuda.stream(stream):
        for _ in range(20):
            busy.add_(1.0)  # the solve runs after the stream's earlier work
    pg.enqueue(**o)
    got, st2 = pg.collect()
    assert np.array_equal(got, want) and st2["iterations"] == st["iterations"]
    assert np.array_equal(pg.pagerank(**o)[0], want)
    pg.set_stream(None)
    pg.close()
