"""The FP32 sweeps over column groups of every width (csrc/sweep.cu: one, two or four pairs of columns, full and partly
filled): a column comes out as it does alone, bit for bit, on trees from one-node leaves to a single front whose inner rows
take several stages.  Needs a GPU."""
import numpy as np
import pytest

from groundtruth_gb300 import native
from test_gpu_small_fronts import _stack
from test_oracle_golden import load

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["small_pair", "small_stack3"])
@pytest.mark.parametrize("leaf", [1, 48, 2000])
@pytest.mark.parametrize("cols", [2, 3, 4, 5, 7, 8, 9, 17])
def test_a_column_does_not_depend_on_its_group(name, leaf, cols):
    z, board = load(name)
    st = _stack(board, leaf)
    obj, k = st.factorise([float(z["op_f"])])[0]
    rng = np.random.default_rng(cols)
    n = st.handle.n_compact
    x = rng.standard_normal((cols, n)) + 1j * rng.standard_normal((cols, n))
    together = native.apply(st.handle, obj, "precond", x, k, "fp32")
    assert np.isfinite(together).all()
    for c in {0, cols // 2, cols - 1}:
        alone = native.apply(st.handle, obj, "precond", x[c], k, "fp32")[0]
        assert np.array_equal(together[c], alone), c
