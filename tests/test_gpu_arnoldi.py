"""The Gram-Schmidt passes that finish in each slot's last block (csrc/gmres.cu: chunk sums, the second pass's decision, the
Givens rotation), at the edges of their chunks (1024 and 2048 unknowns), restart lengths from one step on and with the
second pass never, sometimes and always taken.  Needs a GPU."""
import numpy as np
import pytest

from groundtruth_gb300 import native, stack as gs, synth

pytestmark = pytest.mark.gpu


def _stack(nx, ny):
    d = 0.3e-3
    node = np.ones((nx, ny), bool)
    layers = [synth.Layer("L0", 0.0, 35e-6, node, node[:-1] & node[1:], node[:, :-1] & node[:, 1:])]
    net = synth.Net(synth._segments([(d, d), ((nx - 2) * d, d)], 0.2e-3, 17.5e-6, 0.2e-3), (0, 1, 1), (0, nx - 2, 1))
    return gs.from_board(synth.Board("arnoldi", d, nx, ny, layers, nets=[net], freqs=np.array([1e7])))[0]


# about 290 to 4200 unknowns: one chunk, either side of the chunks' edges, several chunks and a remainder
@pytest.mark.parametrize("nx,ny", [(12, 8), (18, 19), (19, 19), (26, 26), (27, 26), (40, 35)])
@pytest.mark.parametrize("restart,reorth", [(1, 0.7), (2, 0.0), (7, 2.0), (50, 0.0), (50, 0.7), (50, 2.0)])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_solutions_have_their_residual_and_do_not_depend_on_their_neighbours(nx, ny, restart, reorth, precision):
    st = _stack(nx, ny)
    ops = st.factorise([1e7])
    obj, k = ops[0]
    rng = np.random.default_rng(nx * ny)
    cols, n = 3, st.handle.n_compact
    x = rng.standard_normal((cols, n)) + 1j * rng.standard_normal((cols, n))
    b = native.apply(st.handle, obj, "matvec", x, k)
    tol = 1e-9
    opts = dict(tol=tol, restart=restart, max_its=2000, precision=precision, reorth=reorth)
    y, its, res, ok = native.solve(st.handle, ops * cols, b, **opts)
    left = np.linalg.norm(b - native.apply(st.handle, obj, "matvec", y, k), axis=1) / np.linalg.norm(b, axis=1)
    # the reported residual is a recurrence's in FP64, at most 40 updates: it leaves the true one by roundings only
    assert np.all(np.abs(left - res) <= 0.01 * res + 1e-12), (left, res)
    assert its.min() >= 1 and res.max() < 1
    if restart == 50:
        assert ok.all(), (its, res)
    one, its1, _, _ = native.solve(st.handle, ops, b[1:2], **opts)
    assert its1[0] == its[1] and np.array_equal(one[0], y[1])
