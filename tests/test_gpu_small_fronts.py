"""Fronts eliminated and inverted by one CTA each (csrc/factor.cu, small_front_kernel) beside the blocked path, and the FP32
sweeps over the trees they make, at leaf sizes from a few nodes to more rows than a CTA has threads, against the
reference's own preconditioner.  GT_TILED_NF moves fronts between the two: a large value leaves the blocked path only
those that fit no CTA's shared memory.  Needs a GPU."""
import numpy as np
import pytest

from groundtruth_gb300 import native, stack as gs
from test_oracle_golden import load

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def _stack(board, leaf):
    grids = [gs.Grid(0.0, 0.0, board.d * 1e3, board.nx, board.ny, l.node, l.xb, l.yb) for l in board.layers]
    layers = [gs.PlaneLayer(l.name, l.z, g, l.thickness) for l, g in zip(board.layers, grids)]
    return gs.PlaneStack(layers, [gs.Branch(b.a, b.b, b.z, "", b.kind, b.radius) for b in board.branches],
                         [gs.PlanePair(p.upper, p.lower, p.c_per_area, p.tan_delta) for p in board.pairs], board.sigma,
                         precond=board.precond, screen=board.screen, leaf=leaf)


@pytest.mark.parametrize("name", ["small_pair", "small_stack3", "plain_plane"])
@pytest.mark.parametrize("leaf,tiled", [(1, None), (5, 1 << 30), (33, None), (64, 1 << 30), (100, 1 << 30), (200, None),
                                        (2000, 1 << 30)])
def test_preconditioner_matches_the_reference_at_any_leaf_size(name, leaf, tiled, monkeypatch):
    z, board = load(name)
    if tiled:
        monkeypatch.setenv("GT_TILED_NF", str(tiled))
    st = _stack(board, leaf)
    obj, k = st.factorise([float(z["op_f"])])[0]
    y = native.apply(st.handle, obj, "precond", z["prod_x"], k, "fp64")[0]
    assert rel(y, z["prod_precond"]) < 1e-9               # the FP64 preconditioner's tolerance elsewhere
    y32 = native.apply(st.handle, obj, "precond", z["prod_x"], k, "fp32")[0]
    assert rel(y32, z["prod_precond"]) < 1e-3             # and the FP32 sweeps'
