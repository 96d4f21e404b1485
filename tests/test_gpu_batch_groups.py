"""Large batches on large graphs are solved in groups of columns whose results travel
while the next group is solved (two result buffers in turn): the answer of every column
is bit for bit that of the same column in a batch of one group."""

import numpy as np
import pytest

from eggpu_b200 import _native, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("correction", [True, False])
def test_groups_of_columns_match_one_group(pinned, correction):
    g = synth.rmat(scale=16, edgefactor=80, seed=71)
    assert g.m + g.n >= 4 << 20 and g.n * 32 * 8 >= 16 << 20  # the sizes from which groups are used
    pg = _native.PreparedGraph(g.V, g.E)
    sets = synth.seed_sets(g.n, 299, 1, 16, seed=9)  # ten panels, the last one of 11 columns
    o = {"max_iter": 5, "tol": 0.0, "correction": correction}
    out = _native.pinned_empty((299, g.n)) if pinned else np.empty((299, g.n))
    got, st = pg.pagerank_seeds(sets, out=out, **o)
    assert got is out and all(s["iterations"] == 5 for s in st)
    assert len({s["kernel_seconds"] for s in st}) == 1 and st[0]["kernel_seconds"] > 0
    for j0 in range(0, 299, 96):
        part = sets[j0:j0 + 96]
        want, _ = pg.pagerank_seeds(part, **o)
        assert np.array_equal(got[j0:j0 + len(part)], want), j0
    # columns stop on their own rule in every group
    rule, st = pg.pagerank_seeds(sets[:200], max_iter=100, tol=1e-7)
    assert all(s["converged"] for s in st)
    assert np.abs(rule.sum(axis=1) - 1.0).max() < 1e-9
    pg.close()


def test_groups_beside_an_open_session():
    """A batch in groups leaves a session of the same graph alone, and the other way round."""
    g = synth.rmat(scale=16, edgefactor=80, seed=72)
    pg = _native.PreparedGraph(g.V, g.E)
    sets = synth.seed_sets(g.n, 200, 1, 16, seed=10)
    o = {"max_iter": 12, "tol": 0.0}
    want, _ = pg.pagerank_seeds(sets, **o)
    want = want.copy()
    sess = _native.Session(pg, alpha=0.85, tol=0.0, slots=64)
    slots = sess.admit(sets[:40], max_iter=12)
    sess.step(5)
    got, _ = pg.pagerank_seeds(sets, **o)  # while the session's columns are half way
    assert np.array_equal(got, want)
    done = list(sess.step(7))
    assert sorted(done) == sorted(slots)
    ranks, _ = sess.collect(slots)
    assert np.abs(ranks - want[:40]).sum(axis=1).max() <= 1e-12
    sess.close()
    pg.close()
