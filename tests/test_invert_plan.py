"""The steps of the large fronts' selective inversion (csrc/invert_plan.h), compiled on their own with the host compiler: every
front is in each step that it has own columns for, each step's grid reaches its largest front's rows, and the blocks launched are
within four times those with work, on trees of boards up to six planes of 256 x 256.  No GPU."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from groundtruth_gb300 import stack as gs, synth

CSRC = Path(__file__).resolve().parent.parent / "groundtruth_gb300" / "csrc"
SHIM = """
#include "invert_plan.h"
extern "C" int plan(int n, const int64_t* fronts, const int64_t* nown, const int64_t* nbnd, int block, int64_t* order, int* count,
                    int* rows) {
    const gt::InvertPlan P = gt::make_invert_plan(std::vector<int64_t>(fronts, fronts + n), nown, nbnd, block);
    for (int k = 0; k < n; ++k) order[k] = P.fronts[k];
    for (size_t s = 0; s < P.count.size(); ++s) count[s] = P.count[s], rows[s] = P.max_nf[s];
    return (int)P.count.size();
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    cc = shutil.which("g++")
    if not cc:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("invert")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run([cc, "-O1", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", str(d / "shim.cpp"), "-o", str(d / "shim.so")],
                   check=True)
    lib = C.CDLL(str(d / "shim.so"))
    ptr = lambda a, t: a.ctypes.data_as(C.POINTER(t))

    def make(fronts, nown, nbnd):
        fronts, nown, nbnd = (np.ascontiguousarray(a, np.int64) for a in (fronts, nown, nbnd))
        order = np.zeros(max(len(fronts), 1), np.int64)
        count, rows = (np.zeros(int(nown.max(initial=0)) + 1, np.int32) for _ in range(2))
        n = lib.plan(len(fronts), *(ptr(a, C.c_int64) for a in (fronts, nown, nbnd)), 32, ptr(order, C.c_int64),
                     ptr(count, C.c_int), ptr(rows, C.c_int))
        return order[: len(fronts)], count[:n], rows[:n]
    return make


def tiles(rows, kb):
    """Blocks of a step's three launches for a front of that many rows from own column kb on."""
    below = max(0, -(-(rows - kb) // 32))
    return kb // 32 + 1 + below * (-(-kb // 32) + 1)


def _check(plan, nown, nbnd, least):
    fronts = np.flatnonzero(nown + nbnd >= least)
    order, count, rows = plan(fronts, nown, nbnd)
    assert sorted(order) == fronts.tolist()
    launched = needed = 0
    for s in range(len(count)):
        has = nown[order] > 32 * s
        assert has[: count[s]].all() and not has[count[s]:].any()
        nf = (nown + nbnd)[order[: count[s]]]
        assert rows[s] == nf.max()
        launched += count[s] * tiles(int(rows[s]) - 1, 32 * s)
        needed += sum(tiles(int(r) - min(32, int(o) - 32 * s), 32 * s) for r, o in zip(nf, nown[order[: count[s]]]))
    assert not np.any(nown[fronts] > 32 * len(count))
    return launched, needed


@pytest.mark.parametrize("make", [synth.small_pair, lambda: synth.slotted_pair(n=256, n_nets=1, n_freq=1),
                                  lambda: synth.largest_board(256, n_nets=1, n_freq=1)])
def test_steps_have_the_fronts_that_need_them(plan, make):
    sym = gs.from_board(make(), _device=False)[0].sym
    launched, needed = _check(plan, sym.nown, sym.nbnd, 96)
    assert needed <= launched <= 4 * needed


def test_odd_fronts(plan):
    rng = np.random.default_rng(4)
    for _ in range(30):
        n = int(rng.integers(1, 60))
        nown, nbnd = rng.integers(0, 200, n), rng.integers(0, 300, n)
        nown[rng.random(n) < 0.2] = rng.choice([0, 1, 32, 33, 64])
        _check(plan, nown, nbnd, 1)
    assert len(plan([], np.zeros(1), np.zeros(1))[1]) == 0
