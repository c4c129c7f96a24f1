"""Where the 2D sweep's regions and tiles lie (csrc/fi_tile2d_map.h, compiled with the host
compiler): for every side from 3 to 1200 cells, bounded or periodic, and every depth of a
launch, the tiles write each position once, and every value written -- a ghost's source cell
included -- lies at least k layers inside its region.  An iteration makes one more layer at
each edge of a region wrong, so k layers are wrong after a launch of k."""
import ctypes
import os
import subprocess

import pytest

from conftest import ROOT

SOURCE = r"""
#include "fi_tile2d_map.h"
using namespace fi;
// the first side of [3, hi] that breaks a rule for regions of R positions and k iterations, or 0
extern "C" int first_bad(int R, int k, int per, int hi) {
    const int t = R - 2 * k;
    for (int n = 3; n <= hi; n++) {
        const int lo = per ? 1 : 0, end = per ? n : n + 2;
        for (int q = lo; q <= end; q++) {
            int writers = 0;
            for (int b = 0; b < t2_tiles(n, t, per); b++) {
                const int first = 1 + b * t - t2_shift(n, t, per), r0 = first - k;
                if (!t2_owned(q, first, t, n, per)) continue;
                writers++;
                // the position itself (ghosts: the cell that it follows from; n + 2 holds no value)
                const int at[2] = {q == 0 ? 1 : q == n + 2 ? n + 1 : q, n};
                for (int c = 0; c < (q == n + 1 && !per ? 2 : 1); c++)
                    if (at[c] < r0 + k || at[c] > r0 + R - 1 - k) return n;
                if (q < r0 || q > r0 + R - 1) return n;
            }
            if (writers != 1) return n;
        }
    }
    return 0;
}
extern "C" void plan(int n0, int n1, int *shape, int *k) {
    const Tile2DPlan p = tile2d_plan(n0, n1);
    *shape = p.shape, *k = p.k;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("tile2d_map")
    src, out = d / "map.cpp", d / "map.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, "fastice.jl_b200", "csrc"),
                    str(src), "-o", str(out)], check=True)
    return ctypes.CDLL(str(out))


@pytest.mark.parametrize("per", [0, 1], ids=["bounded", "periodic"])
@pytest.mark.parametrize("R,depths", [(32, range(1, 11)), (16, range(1, 7))])
def test_tiles_write_what_their_regions_get_right(lib, R, depths, per):
    bad = {k: n for k in depths if (n := lib.first_bad(R, k, per, 1200))}
    assert not bad, bad


def test_plan_stays_within_the_checked_depths(lib):
    shape, k = ctypes.c_int(), ctypes.c_int()
    seen = set()
    for n0 in range(3, 700, 7):
        for n1 in range(3, 700, 5):
            lib.plan(n0, n1, ctypes.byref(shape), ctypes.byref(k))
            seen.add((shape.value, k.value))
            assert 1 <= k.value <= (6 if shape.value == 0 else 10)
    assert (0, 6) in seen and (0, 5) in seen and (2, 4) in seen
