"""More large fronts than a grid's second dimension holds (65,535; csrc/factor.cu launches them in parts): a plane's tree cut down
to single nodes, every front sent down the blocked path, against the same tree without that.  Needs a GPU."""
import numpy as np
import pytest

from groundtruth_gb300 import native, synth
from test_gpu_small_fronts import _stack, rel

pytestmark = pytest.mark.gpu


def test_more_large_fronts_than_a_grid_is_high(monkeypatch):
    board = synth.plain_plane(n=400)
    ys = []
    for tiled in ("1", str(1 << 30)):
        monkeypatch.setenv("GT_TILED_NF", tiled)
        st = _stack(board, 1)
        assert len(st.sym.nown) > 65535 + 1000
        obj, k = st.factorise([1e8])[0]
        x = np.random.default_rng(1).standard_normal((1, st.handle.n_compact)).astype(np.complex128)
        ys.append([native.apply(st.handle, obj, "precond", x, k, p)[0] for p in ("fp64", "fp32")])
    assert rel(ys[0][0], ys[1][0]) < 1e-9                 # the FP64 preconditioner's tolerance elsewhere
    assert rel(ys[0][1], ys[1][0]) < 1e-3                 # and the FP32 sweeps'
