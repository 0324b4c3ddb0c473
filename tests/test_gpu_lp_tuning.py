"""The launch shapes of the L_p passes that a first product of eight columns times (api.cu, tune_lp): only shapes that differ.
Passes by warps have one of their own, so that their rows or columns per block are not gone through.  Needs a GPU."""
import numpy as np
import pytest

from groundtruth_gb300 import native, stack as gs
from test_sweep_plan import moated

pytestmark = pytest.mark.gpu


# grids whose columns are transformed by warps; with rows of 512 the row passes are too
@pytest.mark.parametrize("nx,ny,rows", [(60, 70, 5), (131, 100, 5), (250, 256, 1)])
def test_a_first_product_times_each_shape_once(nx, ny, rows):
    st, _ = gs.from_board(moated(nx, ny))
    obj, k = st.factorise([1e8])[0]
    rng = np.random.default_rng(nx)
    x = rng.standard_normal((8, st.handle.n_compact)) + 1j * rng.standard_normal((8, st.handle.n_compact))

    def launches():
        n = st.handle.lib.gt_launch_count()
        y = native.apply(st.handle, obj, "matvec", x, k, "fp32")
        return st.handle.lib.gt_launch_count() - n, y
    (first, a), (second, b) = launches(), launches()
    # two orientations, two runs of three passes for each number of rows that a block can take
    assert 0 < first - second <= 2 * rows * 2 * 3
    assert np.array_equal(a, b)
