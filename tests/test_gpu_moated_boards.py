"""Boards whose copper falls apart along a dissection line (a front without a row at the top of a subtree): the FP32
preconditioner, whose sweeps order the pieces by the plan's counters alone, against the FP64 one, whose sweeps go level by
level; several vectors one after the other, so that a piece that was not waited for would show the last vector's.  Needs a
GPU."""
import numpy as np
import pytest

from groundtruth_gb300 import native, stack as gs
from test_gpu_small_fronts import _stack, rel
from test_sweep_plan import moated

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gaps", [((16,), ()), ((16,), (15,)), ((8, 16, 24), ()), ((3,), (29,))])
@pytest.mark.parametrize("leaf", [1, 48])
@pytest.mark.parametrize("cols", [1, 3])
def test_the_preconditioner_of_separate_pieces(gaps, leaf, cols):
    st = _stack(moated(33, 31, *gaps), leaf)
    obj, k = st.factorise([1e8])[0]
    rng = np.random.default_rng(leaf + cols)
    for _ in range(4):
        x = rng.standard_normal((cols, st.handle.n_compact)) + 1j * rng.standard_normal((cols, st.handle.n_compact))
        y32, y64 = (native.apply(st.handle, obj, "precond", x, k, p) for p in ("fp32", "fp64"))
        for c in range(cols):
            assert rel(y32[c], y64[c]) < 1e-3             # the FP32 sweeps' tolerance elsewhere


def test_a_solve_on_one_piece():
    st, routes = gs.from_board(moated(33, 31, (16,), (15,)))
    x = st.solve_batch([1e8], [routes[0].rhs_top(1e8)], [routes[0].J()], tol=1e-10)[0]
    assert x[4] <= 1e-10
