"""The column pass of the FP32 partial-inductance product at every FFT length and sheet count it is built for (warp
transforms of 32 A, csrc/fftw.cuh; the pass's shared-memory multiply), against the FP64 product of the same currents.
Needs a GPU."""
import numpy as np
import pytest

from groundtruth_gb300 import native, stack as gs, synth

pytestmark = pytest.mark.gpu


def _stack(nx, ny, sheets):
    d = 0.3e-3
    layers = []
    for k in range(sheets):
        node = np.ones((nx, ny), bool)
        node[nx // 3: nx // 3 + 2, ny // 4: ny // 2] = k % 2 == 0
        layers.append(synth.Layer(f"L{k}", -k * 0.4e-3, 35e-6, node, node[:-1] & node[1:], node[:, :-1] & node[:, 1:]))
    net = synth.Net(synth._segments([(d, d), ((nx - 2) * d, d)], 0.2e-3, 17.5e-6, 0.2e-3), (0, 1, 1), (0, nx - 2, 1))
    return gs.from_board(synth.Board("lengths", d, nx, ny, layers, nets=[net], freqs=np.array([1e8])))[0]


# (nx, ny, sheets, columns): column lengths 64 to 1024 on either axis, the largest and the smallest grid of a length, rows
# that do not fill the warps, one to six sheets
@pytest.mark.parametrize("nx,ny,sheets,cols", [
    (33, 17, 3, 5), (48, 33, 1, 9), (49, 64, 2, 3), (64, 65, 5, 2), (96, 20, 4, 7), (97, 128, 3, 1), (128, 49, 6, 3),
    (129, 40, 2, 5), (192, 12, 4, 2), (193, 24, 3, 3), (256, 16, 6, 2), (257, 20, 2, 3), (384, 9, 3, 2), (385, 10, 5, 1),
    (512, 8, 2, 2)])
def test_fp32_product_agrees_with_fp64(nx, ny, sheets, cols):
    st = _stack(nx, ny, sheets)
    obj, k = st.factorise([1e8])[0]
    rng = np.random.default_rng(nx * ny)
    x = np.zeros((cols, st.handle.n_compact), complex)
    x[:, : st.ns] = rng.standard_normal((cols, st.ns)) + 1j * rng.standard_normal((cols, st.ns))
    ref = native.apply(st.handle, obj, "lp", x, k, "fp64")[:, : st.ns]
    got = native.apply(st.handle, obj, "lp", x, k, "fp32")[:, : st.ns]
    # two transforms of at most 1024 x 1024 points in FP32: a few times log2(N) roundings of 6e-8, random
    err = np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert err.max() < 2e-6, err
