"""The choice of how many panels of a batch are solved together, on the CPU: few sweeps
hide the read-back behind small groups, many sweeps are solved in large ones, and a
batch is never cut where that is expected to take longer than one group."""

import ctypes
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "eggpu_b200" / "csrc"
MOST = 16  # panels of a launch


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("groups")
    (d / "g.cpp").write_text('#include "batch_groups.h"\nextern "C" int panels(long long e, int n, int p, int s, int m)'
                             '{ return egpr::batch_group_panels(e, n, p, s, m); }\n'
                             'extern "C" int sweeps(double a, double t, int m, int n)'
                             '{ return egpr::expected_sweeps(a, t, m, n); }\n')
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", d / "g.cpp", "-o", d / "g.so"], check=True)
    lib = ctypes.CDLL(str(d / "g.so"))
    lib.panels.argtypes = [ctypes.c_longlong] + [ctypes.c_int] * 4
    lib.sweeps.argtypes = [ctypes.c_double, ctypes.c_double, ctypes.c_int, ctypes.c_int]
    return lib


@pytest.mark.parametrize("entries,n,panels,sweeps,want", [
    (16_500_000, 1 << 20, 8, 20, (2, 3, 4)),  # 256 columns, 20 sweeps: measured best with 3
    (16_500_000, 1 << 20, 8, 100, (6, 7, 8)),
    (16_500_000, 1 << 20, 8, 1000, (8,)),     # nothing to hide the read-back behind is gained
    (9_200_000, 1 << 18, 8, 200, (8,)),       # 18% slower in groups of 3
    (9_200_000, 1 << 18, 4, 50, (4,)),        # 9% slower
    (67_000_000, 1 << 22, 4, 10, (1,)),
])
def test_groups_follow_the_sweeps(lib, entries, n, panels, sweeps, want):
    assert lib.panels(entries, n, panels, sweeps, MOST) in want


@pytest.mark.parametrize("panels", [1, 2, 7, 8, 9, 40, 1000])
def test_groups_stay_in_range(lib, panels):
    for sweeps in (1, 5, 20, 100, 500, 10**6, 2**31 - 1):
        g = lib.panels(16_500_000, 1 << 20, panels, sweeps, MOST)
        assert 1 <= g <= min(panels, MOST)
        assert sweeps < 10**6 or g == min(panels, MOST) or -(-panels // g) == -(-panels // MOST)


def test_expected_sweeps(lib):
    assert lib.sweeps(0.85, 0.0, 77, 1000) == 77
    assert lib.sweeps(0.85, 1e-6, 100, 1 << 20) == 1     # tol * n is about 1
    assert lib.sweeps(0.85, 1e-9, 100, 1 << 20) == 9     # 9 and 16 on R-MAT scale 20
    assert lib.sweeps(0.85, 1e-12, 100, 1 << 20) == 17
    assert lib.sweeps(0.85, 1e-60, 100, 1 << 20) == 100
    assert lib.sweeps(0.85, 1.0, 100, 1 << 20) == 1
    assert lib.sweeps(1.0, 1e-6, 100, 10) == 100 and lib.sweeps(-0.5, 1e-6, 100, 10) == 100
