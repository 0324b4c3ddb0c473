"""gt_moment of more columns than a grid's second dimension takes: the moments of each column by itself, bit for bit.  Needs a
GPU."""
import numpy as np
import pytest

from groundtruth_gb300 import stack as gs
from test_sweep_plan import moated

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [65535, 65536, 131071])
def test_moments_of_many_columns(cols):
    import torch
    st, _ = gs.from_board(moated(5, 4))
    g = torch.Generator(device="cuda").manual_seed(cols)
    x = torch.randn((cols, st.handle.n_dense), dtype=torch.complex128, device="cuda", generator=g)
    torch.cuda.synchronize()
    m = st.handle.moment(cols, x.data_ptr(), st.sheet_z, st.d)
    assert np.isfinite(m).all()
    for c in (0, 1, 65534, cols - 1):
        assert np.array_equal(m[c], st.handle.moment(1, x[c].data_ptr(), st.sheet_z, st.d)[0]), c
