"""Row sums of the two-phase sweep over the values it accepts.  Compared with the FP64
oracle; each tolerance is a bound on FP32 iterates and carried values (24-bit
significands) stated beside it."""

import numpy as np
import pytest

from eggpu_b200 import _native
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
