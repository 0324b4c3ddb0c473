"""The column pass of the FP32 partial-inductance product by warps, with warps that have no rows of their own (few columns: a
small grid, or all columns in one block) and without (many): a column comes out the same bits, at every length and at sheet
counts that leave one to seven helping warps.  Needs a GPU."""
import numpy as np
import pytest

from groundtruth_gb300 import native
from test_gpu_lp_lengths import _stack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(40, 20), (50, 250), (80, 40), (110, 200), (180, 16), (250, 30), (20, 250), (300, 10), (500, 8)])
@pytest.mark.parametrize("sheets", [1, 3, 6])
def test_a_column_alone_and_among_others(nx, ny, sheets):
    st = _stack(nx, ny, sheets)
    obj, k = st.factorise([1e8])[0]
    rng = np.random.default_rng(nx + ny)
    x = np.zeros((33, st.handle.n_compact), complex)
    x[:, : st.ns] = rng.standard_normal((33, st.ns)) + 1j * rng.standard_normal((33, st.ns))
    many = native.apply(st.handle, obj, "lp", x, k, "fp32")
    assert np.isfinite(many).all() and np.any(many)
    for c in (0, 32):
        assert np.array_equal(many[c], native.apply(st.handle, obj, "lp", x[c], k, "fp32")[0])
    assert np.array_equal(many[:2], native.apply(st.handle, obj, "lp", x[:2], k, "fp32"))
    assert not np.any(many[:, st.ns:])                       # (the product is the strips' own)
