"""The system product with its two orientations side by side (small grids) against the same passes one after the other, which
is how the profiler times them: the same kernels on the same values, so the same bits.  Needs a GPU."""
import numpy as np
import pytest

from groundtruth_gb300 import native, stack as gs, synth

pytestmark = pytest.mark.gpu


# grids of 2 x 64 x 32 entries up to either side of 2^20 (S P1 ld0 times the columns), three cells (the least) on either axis
@pytest.mark.parametrize("nx,ny,cols", [(32, 32, 1), (3, 40, 2), (40, 3, 2), (61, 83, 3), (128, 128, 8), (256, 256, 4),
                                        (256, 256, 5)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_the_product_is_the_same_side_by_side(nx, ny, cols, precision):
    d = 0.3e-3
    node = np.ones((nx, ny), bool)
    layers = [synth.Layer(f"L{k}", -k * 0.4e-3, 35e-6, node, node[:-1] & node[1:], node[:, :-1] & node[:, 1:]) for k in range(2)]
    ends = ((0, 0, 0), (0, nx - 1, ny - 1))
    net = synth.Net(synth._segments([(0.0, 0.0), ((nx - 1) * d, (ny - 1) * d)], 0.2e-3, 17.5e-6, 0.2e-3), *ends)
    st = gs.from_board(synth.Board("side", d, nx, ny, layers, nets=[net], freqs=np.array([1e8])))[0]
    obj, k = st.factorise([1e8])[0]
    rng = np.random.default_rng(nx + cols)
    x = rng.standard_normal((cols, st.handle.n_compact)) + 1j * rng.standard_normal((cols, st.handle.n_compact))
    side = [native.apply(st.handle, obj, kind, x, k, precision) for kind in ("matvec", "lp")]
    st.handle.profile(True)
    try:
        turn = [native.apply(st.handle, obj, kind, x, k, precision) for kind in ("matvec", "lp")]
    finally:
        st.handle.profile(False)
    for a, b in zip(side, turn):
        assert np.array_equal(a, b)
        assert np.isfinite(a).all() and np.any(a)
