"""The preparation's radix sort at the key widths where its digits change (8, 9 or 10 bits)
and at the edges of its 4096-item tiles: in_row, in_col and in_w bit for bit as the
reference's stable scatter gives them, with and without dropped destinations."""

import numpy as np
import pytest

from eggpu_b200 import _native
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("dropped", [False, True])
@pytest.mark.parametrize("n,m", [
    (256, 5000), (257, 4095), (512, 4096), (513, 4097), (1024, 12289), (1025, 70000),  # 8 to 11 bits
    ((1 << 17) - 1, 30000), ((1 << 18) + 1, 300001), ((1 << 19) + 1, 8192), (1 << 20, 500000), ((1 << 20) + 1, 65537)])
def test_sorted_entries_match_the_stable_scatter(n, m, dropped, weighted):
    rng = np.random.default_rng(n + m)
    src = np.sort(rng.integers(0, n, m))
    E = np.where(rng.random(m) < 0.3, rng.integers(0, 7, m), rng.integers(0, n, m)).astype(np.int32)
    E[rng.integers(0, m, 5)] = n - 1
    if dropped:
        E[rng.integers(0, m, m // 50)] = n
        E[rng.integers(0, m, m // 50)] = -3
    V = np.zeros(n + 1, np.int32)
    V[1:] = np.cumsum(np.bincount(src, minlength=n))
    W = (1.0 - rng.random(m, np.float32)).astype(np.float64) if weighted else None
    pg = _native.PreparedGraph(V, E, W)
    row, col, w, dangling, outw = pg.export_inbound()
    orow, ocol, ow, odang, ooutw = oracle.build_inbound(V, E, W)
    assert np.array_equal(row, orow) and np.array_equal(col, ocol) and np.array_equal(dangling, odang)
    assert np.array_equal(outw.view(np.uint64), ooutw.view(np.uint64))
    assert np.array_equal(w, ow.astype(np.float32))
    pg.close()
