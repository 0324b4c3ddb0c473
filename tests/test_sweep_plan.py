"""The plan of the FP32 sweeps (csrc/sweep_plan.h): whatever order tasks are let run in by the counters they wait on, a task
finds done what it reads: forward, the boundary rows its children pass up; backward, its front's own forward rows and the
solutions of its boundary rows.  The plan is compiled on its own with the host compiler, on trees of boards whose copper
falls apart along a dissection line among them.  No GPU."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from groundtruth_gb300 import stack as gs, synth

CSRC = Path(__file__).resolve().parent.parent / "groundtruth_gb300" / "csrc"
SHIM = """
#include "sweep_plan.h"
extern "C" int plan(int nf, int nlev, const int64_t* level_ptr, const int64_t* order, const int64_t* own, const int64_t* nown,
                    const int64_t* nbnd, const int64_t* bp, const int64_t* bi, const int64_t* cp, const int64_t* ci,
                    const int64_t* mp, const int64_t* mi, const int64_t* vo, int* out, int cap, int* nft) {
    const gt::SweepPlanHost S = gt::make_sweep_plan(nf, nlev, level_ptr, order, own, nown, nbnd, bp, bi, cp, ci, mp, mi, vo);
    *nft = S.nft;
    for (int t = 0; t < (int)S.tasks.size() && t < cap; ++t) {
        const gt::SwTask& q = S.tasks[t];
        const int v[6] = {q.dep, q.need, q.sig, q.own0, q.r0, q.h};
        for (int k = 0; k < 6; ++k) out[6 * t + k] = v[k];
    }
    return (int)S.tasks.size();
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    cc = shutil.which("g++")
    if not cc:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("plan")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run([cc, "-O1", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", str(d / "shim.cpp"), "-o", str(d / "shim.so")],
                   check=True)
    lib = C.CDLL(str(d / "shim.so"))

    def make(sym):
        arrays = [np.ascontiguousarray(a, np.int64) for a in
                  (sym.level_ptr, sym.order, sym.own_start, sym.nown, sym.nbnd, sym.bnd_ptr, sym.bnd_idx, sym.child_ptr,
                   sym.child_idx, sym.cmap_ptr, sym.cmap_idx, sym.vec_off)]
        args = [a.ctypes.data_as(C.POINTER(C.c_int64)) for a in arrays]
        cap = int((sym.nown + sym.nbnd + sym.nown).sum()) + 1
        out, nft = np.zeros((cap, 6), np.int32), C.c_int(0)
        n = lib.plan(len(sym.nown), len(sym.level_ptr) - 1, *args, out.ctypes.data_as(C.POINTER(C.c_int)), cap, C.byref(nft))
        assert n <= cap
        return out[:n], nft.value
    return make


def moated(nx, ny, gaps_x=(), gaps_y=()):
    """Two planes with the same gaps through both: pieces that nothing joins."""
    d = 0.3e-3
    node = np.ones((nx, ny), bool)
    node[list(gaps_x)] = False
    node[:, list(gaps_y)] = False
    layers = [synth.Layer(f"L{k}", -k * 0.4e-3, 35e-6, node, node[:-1] & node[1:], node[:, :-1] & node[:, 1:])
              for k in range(2)]
    i, j = min([nx, *gaps_x]) - 1, min([ny, *gaps_y]) - 1
    net = synth.Net(synth._segments([(0.0, 0.0), (i * d, j * d)], 0.2e-3, 17.5e-6, 0.2e-3), (0, 0, 0), (0, i, j))
    return synth.Board("moated", d, nx, ny, layers, nets=[net], freqs=np.array([1e8]))


BOARDS = {
    "pair": synth.small_pair, "stack3": synth.small_stack3, "random": lambda: synth.random_board(4),
    "halves": lambda: moated(33, 31, (16,)),                 # the first dissection line is the gap
    "quarters": lambda: moated(33, 31, (16,), (15,)),        # and the lines below it
    "strips": lambda: moated(65, 23, (16, 32, 48)),          # three lines, the middle one first
    "aside": lambda: moated(40, 40, (3,), (29,)),            # gaps that are no dissection line
    "specks": lambda: moated(30, 30, range(2, 30, 3), range(2, 30, 3)),      # pieces of 2 x 2 nodes
}


@pytest.mark.parametrize("name", BOARDS)
@pytest.mark.parametrize("leaf", [1, 6, 48])
def test_what_a_task_reads_is_done_before_it_runs(plan, name, leaf):
    board = BOARDS[name]()
    grids = [gs.Grid(0.0, 0.0, board.d * 1e3, board.nx, board.ny, l.node, l.xb, l.yb) for l in board.layers]
    st = gs.PlaneStack([gs.PlaneLayer(l.name, l.z, g, l.thickness) for l, g in zip(board.layers, grids)],
                       [gs.Branch(b.a, b.b, b.z, "", b.kind, b.radius) for b in board.branches],
                       [gs.PlanePair(p.upper, p.lower, p.c_per_area, p.tan_delta) for p in board.pairs], board.sigma,
                       precond=board.precond, screen=board.screen, leaf=leaf, _device=False)
    sym = st.sym
    tasks, nft = plan(sym)
    nf, front_of = len(sym.nown), np.repeat(np.arange(len(sym.nown)), sym.nown)
    rows = sym.nown + sym.nbnd
    # the tasks' fronts: forward they come by level, each front's tiles covering its rows; backward its own columns
    front = np.empty(len(tasks), int)
    fwd, bwd = [0] * nf, [0] * nf                            # bit sets of each front's tasks
    t = 0
    for back in (False, True):
        order = [f for h in range(len(sym.level_ptr) - 1)[::-1 if back else 1]
                 for f in sym.order[sym.level_ptr[h]: sym.level_ptr[h + 1]]]
        for f in order:
            done, end = 0, int(sym.nown[f] if back else rows[f])
            while done < end:
                assert tasks[t, 4] == done and tasks[t, 5] > 0
                done += tasks[t, 5]
                front[t] = f
                (bwd if back else fwd)[f] |= 1 << t
                t += 1
            assert done == end
    assert t == len(tasks) and nft == sum(b.bit_count() for b in fwd)
    signals = {}
    for t, (_, _, sig, _, _, _) in enumerate(tasks):
        signals.setdefault(int(sig), []).append(t)
    before = [0] * len(tasks)                                # what has finished when a task runs
    for t, (dep, need, _, _, _, _) in enumerate(tasks):
        if need > 0:
            by = signals.get(int(dep), [])
            assert need == len(by) and max(by) < t           # the counter waits for every tile that raises it
            for s in by:
                before[t] |= before[s] | 1 << s
    for t, f in enumerate(front):
        if t < nft:
            reads = sum(fwd[c] for c in sym.child_idx[sym.child_ptr[f]: sym.child_ptr[f + 1]] if sym.nbnd[c])
        else:
            reads = fwd[f]
            for g in set(front_of[sym.bnd_idx[sym.bnd_ptr[f]: sym.bnd_ptr[f + 1]]].tolist()):
                reads |= bwd[g]
        assert reads & ~before[t] == 0, (t, f)
