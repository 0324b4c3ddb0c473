"""gt_operators_bytes against the device memory that operator sets take: what the memory gates admit by.  Trees of one-node
leaves, whose backward tiles are padded, to one front, whose diagonal blocks are inverted.  Needs a GPU."""
import ctypes as C

import pytest

from groundtruth_gb300 import native, synth
from test_gpu_small_fronts import _stack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf", [1, 48, 1 << 20])
@pytest.mark.parametrize("fp32_panels", [False, True])
def test_operators_hold_what_they_are_said_to(leaf, fp32_panels):
    st = _stack(synth.slotted_pair(n=48, n_nets=1, n_freq=1), leaf)
    st.fp32_panels = fp32_panels
    n = 24 if leaf < 1 << 20 else 3
    freqs = [1e6 * (q + 1) for q in range(n)]
    tables = [st._freq_tables(f) for f in freqs]
    free = lambda: native.memory(st.handle, 1)["free"]
    keep = [native.Operators(st.handle, freqs, tables, fp32_panels=fp32_panels)]      # (the first call's own needs)
    before = free()
    keep.append(native.Operators(st.handle, freqs, tables, fp32_panels=fp32_panels))
    took = before - free()
    held, making = st.handle.operators_bytes(n, fp32_panels)
    assert st.resident_bytes(n) == held and st.factorisation_bytes(n) == held + making
    # each of a set's dozen allocations ends on a 2 MiB page, which it may share with others
    assert abs(took - held) <= 13 * (2 << 20), (took, held)
    assert making >= n * 16 * (st.sym.upd_total + (st.sym.panel_total if fp32_panels else 0))


def test_malformed_requests_are_refused():
    lib = native.load()
    assert lib.gt_operators_bytes(None, 1, 0, C.byref(C.c_int64()), None) == native.GT_INVALID_ARGUMENT
