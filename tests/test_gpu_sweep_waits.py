"""Waits of the FP32 sweeps (csrc/sweep.cu) that run out: told to wait a millisecond for a tile that nobody finishes
(GT_SWEEP_TEST_SHORTFALL=1) or for 16 bytes more than a panel stage's copy brings (=2), every kind of call that runs the
sweeps returns GT_TIMEOUT (RuntimeError here) by itself, and the calls after it on the same context are right.  Needs a
GPU."""
import numpy as np
import pytest

from groundtruth_gb300 import native, stack as gs, synth
from test_derived_stacks import branches_of
from test_gpu_small_fronts import _stack, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("short", ["1", "2"])
@pytest.mark.parametrize("leaf", [1, 48, 2000])
@pytest.mark.parametrize("cols", [1, 3, 17])
def test_an_application_reports_it(short, leaf, cols, monkeypatch):
    b = synth.small_stack3()
    st = _stack(b, leaf)
    obj, k = st.factorise([float(b.freqs[0])])[0]
    rng = np.random.default_rng(3)
    x = rng.standard_normal((cols, st.handle.n_compact)) + 1j * rng.standard_normal((cols, st.handle.n_compact))
    monkeypatch.setenv("GT_SWEEP_TEST_SHORTFALL", short)
    with pytest.raises(RuntimeError, match="triangular sweeps ran out"):
        native.apply(st.handle, obj, "precond", x, k, "fp32")
    # a call without sweeps, between the one that ran out and the next, has nothing to report
    ref = native.apply(st.handle, obj, "precond", x, k, "fp64")
    monkeypatch.delenv("GT_SWEEP_TEST_SHORTFALL")
    assert rel(native.apply(st.handle, obj, "precond", x, k, "fp32"), ref) < 1e-3


@pytest.mark.parametrize("precision", ["mixed", "mixed16"])
def test_a_solve_reports_it_and_the_next_is_as_on_a_new_stack(precision, monkeypatch):
    b = synth.small_pair()
    freqs = [float(f) for f in b.freqs]

    def solve(st, routes):
        return st.solve_batch(freqs, [routes[0].rhs_top(f) for f in freqs], [routes[0].J()] * len(freqs), tol=1e-9,
                              precision=precision)
    st, routes = gs.from_board(b)
    st.factorise(freqs, together=True)
    monkeypatch.setenv("GT_SWEEP_TEST_SHORTFALL", "1")
    with pytest.raises(RuntimeError, match="triangular sweeps ran out"):
        solve(st, routes)
    monkeypatch.delenv("GT_SWEEP_TEST_SHORTFALL")
    for a, c in zip(solve(st, routes), solve(*gs.from_board(b))):
        assert a[4] <= 1e-9 and a[2] == c[2] and np.array_equal(a[3], c[3])


def test_a_derived_set_made_by_the_fp32_sweeps_reports_it(monkeypatch):
    """A base whose one front is too large for the FP64 sweeps, so that gt_operators_derive runs the FP32 ones."""
    b = synth.slotted_pair(n=64, n_nets=1, n_freq=1)
    st = _stack(b, 1 << 20)
    assert len(st.sym.nown) == 1 and 2 * int(st.sym.nown[0]) * 16 > 227 * 1024
    dst = st.with_branches(branches_of(synth.what_if_branches(b, seed=5, n_via=2, n_part=1)))
    f = float(b.freqs[0])
    st.factorise([f])
    monkeypatch.setenv("GT_SWEEP_TEST_SHORTFALL", "1")
    with pytest.raises(RuntimeError, match="triangular sweeps ran out"):
        dst.factorise([f])
    monkeypatch.delenv("GT_SWEEP_TEST_SHORTFALL")
    obj, k = dst.factorise([f])[0]
    x = np.ones(dst.handle.n_compact, complex)
    assert np.isfinite(native.apply(dst.handle, obj, "precond", x, k, "fp32")).all()


def test_a_solve_whose_tile_loads_ran_out_reports_it_and_the_next_is_as_on_a_new_stack(monkeypatch):
    """The same for pass C of the FP32 L_p product (GT_LP_TMA_TEST_SHORTFALL), on the smallest board that takes it."""
    b = synth.slotted_pair(n_nets=1, n_freq=1)
    f = float(b.freqs[0])

    def solve(st, routes):
        return st.solve_batch([f], [routes[0].rhs_top(f)], [routes[0].J()], tol=1e-9)[0]
    st, routes = gs.from_board(b)
    st.factorise([f])
    monkeypatch.setenv("GT_LP_TMA_TEST_SHORTFALL", "1")
    with pytest.raises(RuntimeError, match="did not arrive"):
        solve(st, routes)
    monkeypatch.delenv("GT_LP_TMA_TEST_SHORTFALL")
    a, c = solve(st, routes), solve(*gs.from_board(b))
    assert a[4] <= 1e-9 and a[2] == c[2] and np.array_equal(a[3], c[3])
