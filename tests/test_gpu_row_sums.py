"""Row sums of the two-phase sweep over the values it accepts.  Compared with the FP64
oracle; each tolerance is a bound on FP32 iterates and carried values (24-bit
significands) stated beside it."""

import numpy as np
import pytest

from eggpu_b200 import _native, synth
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _sweep_path(monkeypatch):
    monkeypatch.setenv("EGPR_SMALL_NNZ", "0")  # small graphs too take the sweep's path


def _csr(n, src, dst, W=None):
    order = np.lexsort((dst, src))
    V = np.zeros(n + 1, np.int32)
    V[1:] = np.cumsum(np.bincount(src, minlength=n))
    return V, dst[order].astype(np.int32), None if W is None else W[order]


def _random(n, m, seed, weighted=False):
    """A ring (no dangling vertex) and random pairs."""
    rng = np.random.default_rng(seed)
    src = np.concatenate([np.arange(n), rng.integers(0, n, m)])
    dst = np.concatenate([(np.arange(n) + 1) % n, rng.integers(0, n, m)])
    return _csr(n, src, dst, 1.0 - rng.random(n + m) if weighted else None)


def _fading_chain(hops, bulk):
    """Vertices 0..hops in a chain; each also feeds 62 sinks that lead back to vertex 0, so
    a rank falls by 0.85 / 63 per hop.  Beside it a random graph that the chain does not
    reach.  No vertex is dangling: nothing is added to a row far from the seed."""
    u = np.arange(hops)
    sinks = hops + 1 + np.arange(62)
    src = np.concatenate([u, np.repeat(u, 62), [hops], sinks])
    dst = np.concatenate([u + 1, np.tile(sinks, hops), [0], np.zeros(62, int)])
    n0 = hops + 63
    V, E, _ = _random(bulk, 6 * bulk, 3)
    bsrc = np.repeat(np.arange(bulk), np.diff(V))
    return _csr(n0 + bulk, np.concatenate([src, n0 + bsrc]), np.concatenate([dst, n0 + E]))


@pytest.mark.parametrize("correction", [True, False])
@pytest.mark.parametrize("bulk", [64, 60000])
def test_tiny_ranks_keep_their_relative_precision(correction, bulk):
    hops = 19  # down to 2^-119: FP32's normal range
    V, E, W = _fading_chain(hops, bulk)
    n = len(V) - 1
    p = np.zeros(n)
    p[0] = 1.0
    o = {"alpha": 0.85, "max_iter": 60, "tol": 0.0}
    pg = _native.PreparedGraph(V, E, W)
    got, _ = pg.pagerank(personalization=p, correction=correction, **o)
    again, _ = pg.pagerank(personalization=p, correction=correction, **o)
    ref, _, _ = oracle.pagerank_pull(V, E, W, teleport=p, **o)
    chain = slice(0, hops + 1)
    assert ref[hops] < 2.0 ** -115
    # per hop one rounding each of scale, product, sum and rank, 2^-24 at most
    assert (np.abs(got[chain] / ref[chain] - 1.0) <= 4 * (hops + 1) * 2.0 ** -24).all()
    assert np.abs(got - ref).sum() <= 1e-6 and np.array_equal(got, again)
    pg.close()


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("alpha,sweeps", [(-0.5, 12), (1.0, 12), (1.3, 8)])
def test_alpha_outside_the_unit_interval(alpha, sweeps, weighted):
    """The entries accept any alpha; rows may be negative then."""
    graphs = [_random(n, 9 * n, n, weighted) for n in (40013, 3001)]
    pgs = [_native.PreparedGraph(*g) for g in graphs]
    o = {"alpha": alpha, "max_iter": sweeps, "tol": 0.0}
    refs = [oracle.pagerank_pull(*g, **o)[0] for g in graphs]
    p = np.zeros(len(graphs[0][0]) - 1)
    p[[0, 7]] = 0.5
    pref = oracle.pagerank_pull(*graphs[0], teleport=p, **o)[0]

    # four roundings per sweep, each 2^-24 of terms that sum to about 1, and later sweeps
    # multiply them by at most |alpha| each
    bound = 4 * 2.0 ** -24 * sum(abs(alpha) ** j for j in range(sweeps)) * 1.1

    def check(got, ref):
        assert np.abs(got - ref).sum() <= bound

    for correction in (True, False):
        for pg, ref in zip(pgs, refs):
            check(pg.pagerank(correction=correction, **o)[0], ref)
            pg.enqueue(correction=correction, **o)
            got, st = pg.collect()
            check(got, ref)
            assert st["iterations"] == sweeps
        outs, sts = _native.pagerank_multi(pgs, correction=correction, **o)
        for got, ref, st in zip(outs, refs, sts):
            check(got, ref)
            assert st["iterations"] == sweeps
        check(pgs[0].pagerank(personalization=p, correction=correction, **o)[0], pref)
    for pg in pgs:
        pg.close()


@pytest.mark.parametrize("first,second", [(1.2, 0.85), (0.85, 1.2)])
def test_an_enqueued_solve_may_follow_one_of_the_other_path(first, second):
    g = _random(40013, 9 * 40013, 40013)
    pg = _native.PreparedGraph(*g)
    o = {"max_iter": 6, "tol": 0.0}
    pg.enqueue(alpha=first, **o)
    pg.enqueue(alpha=second, **o)
    got, st = pg.collect()
    assert st["iterations"] == 6
    assert np.array_equal(got, pg.pagerank(alpha=second, **o)[0])
    ref, _, _ = oracle.pagerank_pull(*g, alpha=second, **o)
    assert np.abs(got - ref).sum() <= 1e-6
    pg.close()


def test_alpha_outside_the_unit_interval_on_a_large_graph():
    """Small ranks: a row's value is about 2^-21 here, and keeps FP32's relative precision."""
    n, sweeps = (1 << 21) + 5, 3
    V, E, W = _random(n, 9 * n, 5)
    pg = _native.PreparedGraph(V, E, W)
    o = {"alpha": 1.01, "max_iter": sweeps, "tol": 0.0}
    ref, _, _ = oracle.pagerank_pull(V, E, W, **o)
    got, _ = pg.pagerank(correction=False, **o)
    # four roundings per sweep, 2^-24 of a value at most
    assert np.abs(got - ref).sum() <= 4 * sweeps * 2.0 ** -24
    pg.close()


@pytest.mark.parametrize("seed", [1, 2, 3])
@pytest.mark.parametrize("scale,small", [(16, "1000000000"), (18, "0")])
def test_rounding_errors_average_out(monkeypatch, scale, small, seed):
    """Carried values are rounded once, independently: 2^-25 / sqrt(3) = 1.7e-8 rms each, and
    the rows that make up the norm average over a hundred and more sources: 2e-9, bound 4e-9.
    An error shared by all sources of one out-degree would not average (1e-8 was seen)."""
    monkeypatch.setenv("EGPR_SMALL_NNZ", small)  # the one-kernel solve, the sweep
    g = synth.rmat(scale=scale, edgefactor=16, seed=seed)
    o = {"alpha": 0.85, "max_iter": 20, "tol": 0.0}
    pg = _native.PreparedGraph(g.V, g.E)
    got, _ = pg.pagerank(**o)
    ref, _, _ = oracle.pagerank_pull(g.V, g.E, None, **o)
    assert np.linalg.norm(got - ref) <= 4e-9 * np.linalg.norm(ref)
    pg.close()
