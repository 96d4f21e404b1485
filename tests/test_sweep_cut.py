"""The cutting of a plan's tiles into the CTA shares of the sweep's first phase, on the
CPU: a unit that began inside a chunk would drop the open run of the chunk's first part,
so every unit begins on a chunk boundary of its block and ends on one or at the block's
end, the units cover every tile once, and no CTA gets more than its share and a chunk."""

import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "eggpu_b200" / "csrc"
GRID = 148

WRAPPER = r"""
#include "sweep_cut.h"
// One entry per graph in nblocks, shift and cost; block_tile and block_pair one after another.
extern "C" int cut(int count, const int* nblocks, const int* shift, const int* cost, const int* block_tile,
                   const int* block_pair, int grid, int* units, int capacity, int* cta_unit) {
    std::vector<egpr::CutGraph> g;
    for (int i = 0; i < count; ++i) {
        g.push_back({block_tile, block_pair, nblocks[i], shift[i], cost[i]});
        block_tile += nblocks[i] + 1;
        block_pair += nblocks[i] + 1;
    }
    std::vector<egpr::GatherUnit> u;
    std::vector<int32_t> c;
    egpr::cut_gather_units(g.data(), count, grid, u, c);
    if ((int)u.size() > capacity || (int)c.size() != grid + 1) return -1;
    for (size_t i = 0; i < u.size(); ++i) {
        units[4 * i] = u[i].graph;
        units[4 * i + 1] = u[i].block;
        units[4 * i + 2] = u[i].tile0;
        units[4 * i + 3] = u[i].tile1;
    }
    for (int i = 0; i <= grid; ++i) cta_unit[i] = c[i];
    return (int)u.size();
}
"""


@pytest.fixture(scope="module")
def cut(tmp_path_factory):
    d = tmp_path_factory.mktemp("cut")
    (d / "cut.cpp").write_text(WRAPPER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", d / "cut.cpp", "-o", d / "cut.so"], check=True)
    lib = ctypes.CDLL(str(d / "cut.so"))

    def call(graphs, grid=GRID):
        """graphs: (tiles per block, pairs per block, chunk shift, pair cost) each."""
        i32 = lambda a: np.ascontiguousarray(a, np.int32)  # noqa: E731
        ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
        nb, shift, cost = (i32([f(g) for g in graphs]) for f in (lambda g: len(g[0]), lambda g: g[2], lambda g: g[3]))
        bt = [np.concatenate([[0], np.cumsum(g[0])]) for g in graphs]
        bp = [np.concatenate([[0], np.cumsum(g[1])]) for g in graphs]
        t, p = i32(np.concatenate(bt)), i32(np.concatenate(bp))
        units, ctas = np.zeros((int(nb.sum()) + grid + 8, 4), np.int32), np.zeros(grid + 1, np.int32)
        k = lib.cut(len(graphs), ptr(nb), ptr(shift), ptr(cost), ptr(t), ptr(p), grid, ptr(units), len(units), ptr(ctas))
        assert k >= 0
        return units[:k], ctas, bt, bp

    return call


def _check(graphs, units, ctas, bt, bp, grid=GRID):
    first = np.concatenate([[0], np.cumsum([b[-1] for b in bt])])
    at = 0  # next tile, counted over all graphs
    cost = np.zeros(len(units))
    for j, (g, b, t0, t1) in enumerate(units):
        chunk = 1 << graphs[g][2]
        b0, b1 = bt[g][b], bt[g][b + 1]
        assert b0 <= t0 < t1 <= b1 and first[g] + t0 == at
        assert (t0 - b0) % chunk == 0 and ((t1 - b0) % chunk == 0 or t1 == b1), (j, g, b, t0 - b0, t1 - t0, b1 - b0)
        at = first[g] + t1
        cost[j] = (t1 - t0) * (256 + graphs[g][3] * (bp[g][b + 1] - bp[g][b]) / (b1 - b0))
    assert at == first[-1]
    assert ctas[0] == 0 and ctas[-1] == len(units) and (np.diff(ctas) >= 0).all()
    share, chunk = cost.sum() / grid, max((1 << g[2]) * (256 * (1 + g[3])) for g in graphs)
    assert max(cost[a:b].sum() for a, b in zip(ctas[:-1], ctas[1:])) <= share + 2 * chunk


@pytest.mark.parametrize("nblocks,tiles", [(1, 10000), (2, 40000), (67, 64500), (110, 256000), (630, 2100000)])
@pytest.mark.parametrize("shift", [0, 2])
def test_units_keep_to_chunks(cut, nblocks, tiles, shift):
    rng = np.random.default_rng(nblocks * 8 + shift)
    for _ in range(100 if nblocks < 200 else 10):
        share = rng.pareto(1.2, nblocks) + 0.2
        t = np.maximum(1, (share / share.sum() * tiles).astype(int))
        g = [(t, rng.integers(t, 256 * t + 1), shift, int(rng.choice([0, 1, 2, 4, 7, 8, 64])))]
        _check(g, *cut(g))


@pytest.mark.parametrize("cost", [0, 4])
@pytest.mark.parametrize("extra", [0, 1, 3, 4])
def test_equal_blocks_that_divide_the_grid(cut, cost, extra):
    for per_cta in (4, 12, 100, 436):
        for nblocks in (1, 4, 37, 74, 148):
            t = np.full(nblocks, per_cta * GRID // nblocks)
            t[-1] += extra
            g = [(t, 50 * t, 2, cost)]
            _check(g, *cut(g))


def test_several_graphs_in_one_plan(cut):
    rng = np.random.default_rng(11)
    for _ in range(50):
        g = []
        for _ in range(int(rng.integers(2, 9))):
            t = rng.integers(1, 9000, int(rng.integers(1, 30)))
            g.append((t, rng.integers(t, 200 * t), int(rng.choice([0, 2])), 4))
        _check(g, *cut(g))


@pytest.mark.parametrize("grid", [1, 2, 148])
def test_few_tiles(cut, grid):
    for tiles in (1, 2, 3, 4, 5, 147, 148, 149):
        for shift in (0, 2):
            g = [([tiles], [3 * tiles], shift, 4)]
            _check(g, *cut(g, grid), grid=grid)
