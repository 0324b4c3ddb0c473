"""The work that users of this package give it, as cases to be timed and compared.

A case is one call (or the few calls that belong together) of the solver's public entry points on a seeded synthetic
board:

    solve    columns K x = b to a tolerance: from host buffers (native.solve, what RouteExcitation.solve ends in) or
             device-resident (Geometry.solve_device, what a batched sweep or a server keeps on the card)
    factor   the Schur complements of a set of frequencies factorised (native.Operators) and the preconditioner they
             make applied once to a vector per frequency (native.apply)
    matvec   the FP64 system product of a few vectors from host buffers (native.apply: the warm start's products)
    lp       the partial-inductance product of device-resident strip currents (gt_lp_product_noalloc)
    fields   the node fields and moments of device-resident solutions (Geometry.node_field, Geometry.moment)
    psi      a signal path's coupling to every strip (Geometry.strip_coupling)

Boards: "plane" one solid plane, "pair" a slotted ground plane over a power plane (preconditioner "sheet") with `parts`
decoupling capacitors between them, "stack" two to five planes of unequal sides with cut-outs and stitching vias
(preconditioner "diag").  A factorisation of a pair always has parts: a plane held by its capacitance alone makes a pivot
so small that its rounding, and nothing else, would be compared.  Solves stop at 1e-12,
tighter than a board's usual 1e-10, so that solutions reached through another order of FP32 roundings agree."""
import ctypes
import math

import numpy as np
import torch

from groundtruth_gb300 import native, stack, synth

TOL = 1e-12


def listed():
    return [
        # one net at one frequency on a small board, as an interactive check asks for it: latency and launches
        dict(name="solve-small", kind="solve", board="pair", nx=32, ny=32, nets=1, freqs=1, host=True, reorth=0.7),
        # the CPU-runnable size: one plane, one net, one frequency, host buffers in and out
        dict(name="solve-plane", kind="solve", board="plane", nx=96, ny=96, nets=1, freqs=1, host=True, reorth=0.7),
        # a ragged four-plane board of an uneven batch, a few nets at a few frequencies, the default options
        dict(name="solve-stack", kind="solve", board="stack", nx=131, ny=203, layers=4, nets=2, freqs=3, host=False,
             reorth=0.7),
        # the benchmark's board and options, a share of its sweep (all its nets at four frequencies)
        dict(name="solve-sweep", kind="solve", board="pair", nx=256, ny=256, nets=8, freqs=4, host=False, reorth=0.0),
        # factorisations: a small three-plane board, a ragged one, the benchmark's board with decoupling parts, as a
        # what-if service holds it, at four of its frequencies
        dict(name="factor-small", kind="factor", board="stack", nx=44, ny=61, layers=3, freqs=2),
        dict(name="factor-stack", kind="factor", board="stack", nx=143, ny=97, layers=4, freqs=3),
        dict(name="factor-sweep", kind="factor", board="pair", nx=256, ny=256, parts=8, freqs=4),
        # the warm start of four columns on the benchmark's board
        dict(name="matvec-warm", kind="matvec", board="pair", nx=256, ny=256, cols=4),
        # products of device-resident currents: one column of a ragged board, a batch on the benchmark's board
        dict(name="lp-ragged", kind="lp", board="stack", nx=83, ny=61, layers=3, cols=1),
        dict(name="lp-batch", kind="lp", board="pair", nx=256, ny=256, cols=8),
        # the maps and moments of a solved batch
        dict(name="fields-batch", kind="fields", board="pair", nx=256, ny=256, cols=32),
        # a net's coupling, made once per net
        dict(name="psi-net", kind="psi", board="pair", nx=256, ny=256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "factor", "factor", "matvec", "lp", "lp", "fields", "psi"])
    board = rng.choice(["pair", "stack"])
    case = dict(kind=kind, board=board)
    if board == "pair":
        case["nx"] = case["ny"] = _log_int(rng, 32, 256)
        case["parts"] = rng.randint(2, 8) if kind == "factor" else rng.choice([0, 0, 4])
        sheets = 2
    else:
        case["nx"], case["ny"] = _log_int(rng, 30, 200), _log_int(rng, 30, 200)
        sheets = case["layers"] = rng.randint(2, 5)
    nodes = sheets * case["nx"] * case["ny"]
    most = 2 * 256 * 256                      # nodes of the largest listed board
    if kind == "solve":
        case.update(nets=rng.randint(1, 4), freqs=rng.randint(1, 4), host=rng.random() < 0.5, reorth=rng.choice([0.0, 0.7]))
        while case["nets"] * case["freqs"] * nodes > 8 * most:
            case["freqs"] = max(1, case["freqs"] - 1)
            case["nets"] = max(1, case["nets"] - (case["freqs"] == 1))
            if case["nets"] == case["freqs"] == 1:
                break
    elif kind == "factor":
        case.update(freqs=max(1, min(4, _log_int(rng, 1, 5) * most // (2 * nodes) or 1)))
    elif kind == "matvec":
        case.update(cols=max(1, min(_log_int(rng, 1, 16), 3 * most // nodes)))
    elif kind == "lp":
        case.update(cols=max(1, min(_log_int(rng, 1, 16), 3 * most // nodes)))
    elif kind == "fields":
        case.update(cols=max(1, min(_log_int(rng, 1, 64), 32 * most // nodes)))
    return case


# ------------------------------------------------------------------------------------------ boards
def _stack_board(nx, ny, layers, nets, rng):
    """Planes nx x ny at 0.3 mm with polygon cut-outs, vias that stitch neighbours, and traces over the top plane whose
    return vias stand in its border (clear of the cut-outs)."""
    d, t = 0.3e-3, 35e-6
    w, h = (nx - 1) * d, (ny - 1) * d
    outline = np.array([[-d / 2, -d / 2], [w + d / 2, -d / 2], [w + d / 2, h + d / 2], [-d / 2, h + d / 2]])
    z, planes = 0.0, []
    for k in range(layers):
        cuts = []
        for _ in range(int(rng.integers(1, 5))):
            c = np.array([rng.uniform(0.25, 0.75) * w, rng.uniform(0.25, 0.75) * h])
            ang = np.sort(rng.uniform(0, 2 * math.pi, int(rng.integers(3, 9))))
            rad = rng.uniform(0.03, 0.09, len(ang)) * min(w, h)
            cuts.append(c + np.stack([rad * np.cos(ang), rad * np.sin(ang)], 1))
        planes.append(synth.Layer("L%d" % k, z, t, *synth.raster_layer(nx, ny, d, outline, cuts)))
        z -= float(rng.uniform(0.1, 1.5)) * 1e-3 + t
    vias = []
    for k in range(layers - 1):
        length = planes[k].z - planes[k + 1].z
        for _ in range(int(rng.integers(2, 9))):
            i, j = int(rng.integers(1, nx - 1)), int(rng.integers(1, ny - 1))
            if planes[k].node[i, j] and planes[k + 1].node[i, j]:
                r = length / (synth.SIGMA_CU * math.pi * 2 * 1.5e-4 * 25e-6)
                vias.append(synth.BranchSpec((k, i, j), (k + 1, i, j), r, 2e-7 * length, 0.0, "via", 1.5e-4))
    z_face, z_sig = t / 2, 0.15e-3 + t
    loops = []
    for _ in range(nets):
        # from the left border over an L-shaped walk to the right border
        a = (int(rng.integers(1, max(2, nx // 10))), int(rng.integers(ny // 8, ny - ny // 8)))
        b = (nx - 1 - int(rng.integers(1, max(2, nx // 10))), int(rng.integers(ny // 8, ny - ny // 8)))
        m = (int(rng.integers(nx // 3, 2 * nx // 3)), a[1])
        pts = [np.array(p) * d for p in (a, m, (m[0], b[1]), b)]
        rows = [[*pts[0], z_face, *pts[0], z_sig, 0.15e-3, 1.0]]
        rows += [[*p, z_sig, *q, z_sig, 0.15e-3, 1.0] for p, q in zip(pts[:-1], pts[1:]) if np.any(p != q)]
        rows += [[*pts[-1], z_sig, *pts[-1], z_face, 0.15e-3, 1.0]]
        loops.append(synth.Net(np.array(rows, float), (0, *a), (0, *b)))
    return synth.Board("stack", d, nx, ny, planes, [], vias, loops, precond="diag")


def _pair_board(n, nets, seed, parts=0):
    b = synth.slotted_pair(n, 0.25 * 256 / max(n, 64), n_nets=nets, n_freq=1, seed=seed,
                           seg_range=(20, 60) if n >= 128 else (6, 14))
    rng = np.random.default_rng([n, parts])
    while len(b.branches) < parts:
        i, j = int(rng.integers(2, n - 2)), int(rng.integers(2, n - 2))
        if b.layers[0].node[i, j]:
            b.branches.append(synth.BranchSpec((0, i, j), (1, i, j), 0.02, 0.5e-9, 100e-9, "part"))
    return b


def _board(case):
    """The case's board, the same for every seed: what changes from call to call are the frequencies, vectors and
    traces that a program brings to a board it holds."""
    if case["board"] == "plane":
        return synth.plain_plane(case["nx"])
    if case["board"] == "pair":
        return _pair_board(case["nx"], case.get("nets", 1), 2, case.get("parts", 0))
    rng = np.random.default_rng([case["nx"], case["ny"], case["layers"]])
    return _stack_board(case["nx"], case["ny"], case["layers"], case.get("nets", 1), rng)


def _rng(seed):
    return np.random.default_rng([seed, 77])


def _freqs(rng, k):
    """k frequencies spread over 1 MHz - 1 GHz, one in each share of the band."""
    return [float(10 ** (6 + 3 * (q + rng.uniform(0.1, 0.9)) / k)) for q in range(k)]


def _vectors(n, cols, seed, mask=None):
    """Complex columns of unit-size random entries (the spread of a Krylov vector's), zero where mask is."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((cols, n), dtype=torch.complex128, device="cuda", generator=g)
    return x if mask is None else x * torch.as_tensor(mask, device="cuda")


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def prepare(case, seed):
    rng = _rng(seed)
    board = _board(case)
    kind = case["kind"]
    st, routes = stack.from_board(board)
    geo = st.handle
    s = dict(kind=kind, st=st, geo=geo, board=board)
    if kind == "solve":
        freqs = _freqs(rng, case["freqs"])
        ops = st.factorise(freqs, together=True)
        cols = [(r, q) for r in range(len(routes)) for q in range(len(freqs))]
        rhs = np.stack([st.rhs_vector(routes[r].rhs_top(freqs[q]), routes[r].J()) for r, q in cols])
        s.update(freqs=freqs, cols=cols, host=case["host"], reorth=case["reorth"])
        if case["host"]:
            s.update(rhs=rhs, ops=[ops[q] for _, q in cols])
        else:
            s["obj"], s["op"] = ops[0][0], np.array([ops[q][1] for _, q in cols], np.int32)
            s["rhs"] = torch.zeros((len(cols), geo.n_dense), dtype=torch.complex128, device="cuda")
            s["x"] = torch.zeros_like(s["rhs"])
            geo.to_dense(rhs, s["rhs"].data_ptr())
            torch.cuda.synchronize()
    elif kind in ("factor", "matvec"):
        n, k = geo.n_compact, case.get("freqs", 1)
        s["freqs"] = [stack.freq_key(f) for f in _freqs(rng, k)]
        s["tables"] = [st._freq_tables(f) for f in s["freqs"]]
        c = case.get("cols", k)
        s["op"] = np.arange(c, dtype=np.int32) if kind == "factor" else np.zeros(c, np.int32)
        s["v"] = rng.standard_normal((c, n)) + 1j * rng.standard_normal((c, n))
        if kind == "matvec":
            # a capacitance's current is its voltage over its impedance, as in a solution
            s["v"][:, st.ns: st.ns + st.ncap] /= max(1.0, float(np.abs(s["tables"][0][2]).max(initial=0.0)))
            s["ops"] = native.Operators(geo, s["freqs"], s["tables"])
    elif kind in ("lp", "fields"):
        s["x"] = _vectors(geo.n_dense, case["cols"], seed, st.dense.mask.astype(np.float64))
        if kind == "lp":
            s["y"] = torch.zeros_like(s["x"])
        else:
            s["kx"] = torch.zeros((case["cols"], st.N, st.nx, st.ny), dtype=torch.complex128, device="cuda")
            s["ky"] = torch.zeros_like(s["kx"])
    elif kind == "psi":
        # a trace drawn like the boards' own
        if case["board"] == "pair":
            s["segments"] = _pair_board(case["nx"], 1, 3 + seed % 100003).nets[0].segments
        else:
            s["segments"] = _stack_board(case["nx"], case["ny"], 1, 1, rng).nets[0].segments
    return s


def run(s):
    kind, geo, st = s["kind"], s["geo"], s["st"]
    if kind == "solve":
        if s["host"]:
            return native.solve(geo, s["ops"], s["rhs"], tol=TOL, reorth=s["reorth"])[0]
        geo.solve_device(s["obj"], s["op"], s["rhs"].data_ptr(), s["x"].data_ptr(), tol=TOL, reorth=s["reorth"],
                         stream=torch.cuda.current_stream().cuda_stream)
        return s["x"]
    if kind == "factor":
        ops = native.Operators(geo, s["freqs"], s["tables"])
        return native.apply(geo, ops, "precond", s["v"], s["op"], "fp64")
    if kind == "matvec":
        return native.apply(geo, s["ops"], "matvec", s["v"], s["op"], "fp64")
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "lp":
        rc = geo.lib.gt_lp_product_noalloc(geo.h, len(s["x"]), _ptr(s["x"]), _ptr(s["y"]), ctypes.c_void_p(stream))
        if rc != native.GT_OK:
            raise RuntimeError(geo.lib.gt_last_error())
        return s["y"]
    if kind == "fields":
        geo.node_field(len(s["x"]), s["x"].data_ptr(), st.d, s["kx"].data_ptr(), s["ky"].data_ptr(), stream)
        m = geo.moment(len(s["x"]), s["x"].data_ptr(), st.sheet_z, st.d, stream)
        return s["kx"], s["ky"], m
    return geo.strip_coupling(st.sheet_z, st.sheet_t, st.d, s["segments"], st.ns)


# ------------------------------------------------------------------------------------------ what a pass cannot do without
def _sizes(case):
    """(sheets, x strips, y strips, capacitance cells, nodes) of a full board of these sides."""
    sheets = {"plane": 1, "pair": 2}.get(case["board"], case.get("layers", 1))
    nx, ny = case["nx"], case["ny"]
    return sheets, sheets * (nx - 1) * ny, sheets * nx * (ny - 1), nx * ny if case["board"] == "pair" else 0, sheets * nx * ny


def _fft_flops(case):
    """The L_p product of one column: forward and inverse transforms of every sheet over both orientations' padded
    grids (5 N log2 N) and the sheet by sheet multiply."""
    sheets, nx, ny = _sizes(case)[0], case["nx"], case["ny"]
    total = 0.0
    for a, b in ((nx - 1, ny), (nx, ny - 1)):
        n = (2 * a - 1) * (2 * b - 1)
        total += 2 * sheets * 5 * n * math.log2(n) + 4 * sheets * sheets * n
    return total


def work(case):
    kind = case["kind"]
    sheets, xs, ys, caps, nodes = _sizes(case)
    n = xs + ys + caps + nodes
    spectra = 8 * sheets * sheets * 2 * case["nx"] * case["ny"]
    # a planar separator tree's factor: ~8 N log2 N entries and ~40 N^1.5 multiply-adds for N nodes in each sheet coupled
    # at every position
    grid = case["nx"] * case["ny"]
    factor_entries = sheets * sheets * 4 * grid * math.log2(grid)
    factor_flops = 8 * sheets ** 3 * 10 * grid ** 1.5
    if kind == "solve":
        cols, its = case["nets"] * case["freqs"], 100
        # per iteration and column in FP32: the product, the preconditioner's sweeps, the projections onto ~25 vectors
        flops = cols * its * (_fft_flops(case) + 16 * factor_entries + 2 * 25 * 8 * n)
        per_it = 8 * (2 * 25 + 6) * n
        return dict(bytes=cols * 32 * n + its * (cols * per_it + case["freqs"] * 16 * factor_entries), flops=flops)
    if kind == "factor":
        return dict(bytes=case["freqs"] * (48 * factor_entries + 32 * n), flops=case["freqs"] * factor_flops)
    if kind == "matvec":
        return dict(bytes=case["cols"] * 32 * n + spectra, flops=case["cols"] * (_fft_flops(case) + 20 * n))
    if kind == "lp":
        return dict(bytes=case["cols"] * 32 * (xs + ys) + spectra, flops=case["cols"] * _fft_flops(case))
    if kind == "fields":
        return dict(bytes=case["cols"] * (32 * (xs + ys) + 16 * caps + 32 * nodes), flops=case["cols"] * 14 * n)
    return dict(bytes=8.0 * (xs + ys), flops=40.0 * 100 * (xs + ys) * 0.5)


# ------------------------------------------------------------------------------------------ in 64 bits, with torch alone
def _dense_convolve(s, strips):
    """L_p times strip currents (cols, X | Y over the full grids): the spectra's circular convolution by torch.fft."""
    st = s["st"]
    S, nx, ny = st.n_sheets, st.nx, st.ny
    out = []
    for o, (n0, n1), x in (("x", (nx - 1, ny), strips[0]), ("y", (nx, ny - 1), strips[1])):
        P0, P1 = st.P[o]
        q = torch.as_tensor(st.spectrum[o], device="cuda") * (P0 * P1)              # (Q1, Q0, S, S)
        i0 = torch.arange(P0, device="cuda")
        i1 = torch.arange(P1, device="cuda")
        full = q[torch.minimum(i1, P1 - i1)][:, torch.minimum(i0, P0 - i0)]         # (P1, P0, S, S)
        y = torch.empty_like(x)
        for c in range(x.shape[0]):
            f = torch.fft.fft2(x[c], s=(P0, P1))                                    # (S, P0, P1)
            y[c] = torch.fft.ifft2(torch.einsum("qpst,tpq->spq", full.to(f.dtype), f))[:, :n0, :n1]
        out.append(y)
    return out


def _strip_grids(s, dense):
    st = s["st"]
    D, S, nx, ny = st.dense, st.n_sheets, st.nx, st.ny
    c = dense.shape[0]
    nX, nY = S * (nx - 1) * ny, S * nx * (ny - 1)
    return (dense[:, D.off_x: D.off_x + nX].reshape(c, S, nx - 1, ny),
            dense[:, D.off_y: D.off_y + nY].reshape(c, S, nx, ny - 1))


def _incidence(s):
    """Ar of strips, capacitances and branches on the kept nodes as (rows, cols, signs), and the kept nodes' count."""
    t = s["st"].top
    kept = -np.ones(t.n_nodes, np.int64)
    kept[t.keep] = np.arange(int(t.keep.sum()))
    nid = t.nid
    a = [nid[t.xa[:, 0], t.xa[:, 1], t.xa[:, 2]], nid[t.ya[:, 0], t.ya[:, 1], t.ya[:, 2]]]
    b = [nid[t.xa[:, 0], t.xa[:, 1] + 1, t.xa[:, 2]], nid[t.ya[:, 0], t.ya[:, 1], t.ya[:, 2] + 1]]
    if len(t.cap):
        u = t.cap[:, :4].astype(np.int64)
        a.append(nid[u[:, 0], u[:, 2], u[:, 3]])
        b.append(nid[u[:, 1], u[:, 2], u[:, 3]])
    if t.nbr:
        a.append(t.branch_ab[:, 0])
        b.append(t.branch_ab[:, 1])
    a, b = kept[np.concatenate(a)], kept[np.concatenate(b)]
    row = np.arange(len(a))
    rows = np.concatenate([row[a >= 0], row[b >= 0]])
    cols = np.concatenate([a[a >= 0], b[b >= 0]])
    sign = np.concatenate([np.ones(int((a >= 0).sum())), -np.ones(int((b >= 0).sum()))])
    return rows, cols, sign, int(t.keep.sum())


def _sparse(rows, cols, vals, shape):
    idx = torch.as_tensor(np.stack([rows, cols]), device="cuda")
    return torch.sparse_coo_tensor(idx, torch.as_tensor(np.asarray(vals, np.complex128), device="cuda"), shape).coalesce()


def _impedances(s, q):
    """(omega, per strip the sheet's impedance, then the capacitances' and the branches' own) at frequency q."""
    w, zs, zcap, zbr, _ = s["tables"][q]
    t = s["st"].top
    pair = np.concatenate([np.full(int(t.cap_mask[p].sum()), p) for p in range(len(t.pair_layers))]) if len(t.cap) else []
    z = np.concatenate([zs[t.xa[:, 0]], zs[t.ya[:, 0]], zcap[np.asarray(pair, np.int64)] if len(t.cap) else [], zbr])
    return w, torch.as_tensor(z.astype(np.complex128), device="cuda")


def _exact_system(s, x, q):
    """K x of compact columns x at frequency q."""
    st = s["st"]
    t, n, nb = st.top, st.handle.n_compact, st.nb
    c2d = torch.as_tensor(st.dense.compact_to_dense, device="cuda")
    dense = torch.zeros((x.shape[0], st.handle.n_dense), dtype=torch.complex128, device="cuda")
    dense[:, c2d] = x
    lx, ly = _dense_convolve(s, _strip_grids(s, dense))
    flux = torch.zeros_like(dense)
    D = st.dense
    flux[:, D.off_x: D.off_x + lx[0].numel()] = lx.reshape(len(x), -1)
    flux[:, D.off_y: D.off_y + ly[0].numel()] = ly.reshape(len(x), -1)
    w, z = _impedances(s, q)
    rows, cols, sign, kept = _incidence(s)
    A = _sparse(rows, cols, sign, (nb, kept))
    I, V = x[:, :nb], x[:, nb:]
    top = z * I - (A @ V.T).T
    top[:, : t.ns] += 1j * w * flux[:, c2d[: t.ns]]
    return torch.cat([top, (A.t() @ I.T).T], 1)


def _exact_precond(s, v, q):
    """[D^-1 (r + Ar y); y] with y = S^-1 (r_V - Ar^T D^-1 r), S dense."""
    st = s["st"]
    t, nb, S = st.top, st.nb, st.n_sheets
    tab = s["tables"][q][4]
    ncode = 1 << S
    r, c, val = [], [], []
    for o, idx, lo in ((0, t.xa, 0), (1, t.ya, t.nxb)):
        code = st.code["xy"[o]][idx[:, 1], idx[:, 2]].astype(np.int64)
        at = -np.ones((S, *st.code["xy"[o]].shape), np.int64)
        at[tuple(idx.T)] = lo + np.arange(len(idx))
        for l in range(S):
            other = at[l, idx[:, 1], idx[:, 2]]
            e = tab[((o * ncode + code) * S + idx[:, 0]) * S + l]
            ok = (other >= 0) & (e != 0)
            r.append(lo + np.flatnonzero(ok)); c.append(other[ok]); val.append(e[ok])
    pair = np.concatenate([np.full(int(t.cap_mask[p].sum()), p) for p in range(len(t.pair_layers))]) if len(t.cap) else np.zeros(0)
    tail = np.concatenate([tab[st.tab_cap0 + pair.astype(np.int64)], tab[st.tab_br0:]])
    r.append(t.ns + np.arange(len(tail))); c.append(t.ns + np.arange(len(tail))); val.append(tail)
    Di = _sparse(np.concatenate(r), np.concatenate(c), np.concatenate(val), (nb, nb))
    rows, cols, sign, kept = _incidence(s)
    A = _sparse(rows, cols, sign, (nb, kept))
    Sc = torch.sparse.mm(A.t(), torch.sparse.mm(Di, A)).to_dense()
    r1 = v[:nb, None]
    y = torch.linalg.solve(Sc, v[nb:, None] - A.t() @ (Di @ r1))
    return torch.cat([Di @ (r1 + A @ y), y])[:, 0]


def _dense_system(s, q):
    """K as a dense matrix, column block by column block."""
    n = s["geo"].n_compact
    K = torch.empty((n, n), dtype=torch.complex128, device="cuda")
    for c0 in range(0, n, 512):
        e = torch.zeros((min(512, n - c0), n), dtype=torch.complex128, device="cuda")
        e[torch.arange(len(e)), c0 + torch.arange(len(e))] = 1
        K[:, c0: c0 + len(e)] = _exact_system(s, e, q).T
    return K


def exact(case, seed):
    kind = case["kind"]
    nodes = _sizes(case)[4]
    if kind == "solve":
        if nodes > 2100 or not case["host"]:
            return None                    # a dense solve of more than ~7000 unknowns
        s = prepare(case, seed)
        s["tables"] = [s["st"]._freq_tables(stack.freq_key(f)) for f in s["freqs"]]
        out = torch.zeros((len(s["cols"]), s["geo"].n_compact), dtype=torch.complex128, device="cuda")
        for q in range(len(s["freqs"])):
            sel = [c for c, (_, k) in enumerate(s["cols"]) if k == q]
            b = torch.as_tensor(s["rhs"][sel], device="cuda")
            K = _dense_system(s, q)
            x = torch.linalg.solve(K, b.T)
            x = x + torch.linalg.solve(K, b.T - K @ x)
            out[sel] = x.T
        return out.cpu().numpy()
    if kind == "factor" and nodes > 9000:
        return None
    s = prepare(case, seed)
    st = s["st"]
    if kind == "factor":
        return torch.stack([_exact_precond(s, torch.as_tensor(s["v"][q], device="cuda"), q) for q in range(len(s["freqs"]))]).cpu().numpy()
    if kind == "matvec":
        return _exact_system(s, torch.as_tensor(s["v"], device="cuda"), 0).cpu().numpy()
    if kind == "lp":
        lx, ly = _dense_convolve(s, _strip_grids(s, s["x"]))
        D, y = st.dense, torch.zeros_like(s["x"])
        y[:, D.off_x: D.off_x + lx[0].numel()] = lx.reshape(len(lx), -1)
        y[:, D.off_y: D.off_y + ly[0].numel()] = ly.reshape(len(ly), -1)
        return y * torch.as_tensor(D.mask.astype(np.float64), device="cuda")
    if kind == "fields":
        return _exact_fields(s)
    return _exact_psi(s)


def _exact_fields(s):
    st, x, d = s["st"], s["x"], s["st"].d
    X, Y = _strip_grids(s, x)
    kx, ky = torch.zeros_like(s["kx"]), torch.zeros_like(s["ky"])
    cx, cy = torch.zeros(kx.shape, device="cuda", dtype=torch.float64), torch.zeros(kx.shape, device="cuda", dtype=torch.float64)
    kx[:, :, :-1] += X
    kx[:, :, 1:] += X
    cx[:, :, :-1] += X != 0
    cx[:, :, 1:] += X != 0
    ky[:, :, :, :-1] += Y
    ky[:, :, :, 1:] += Y
    cy[:, :, :, :-1] += Y != 0
    cy[:, :, :, 1:] += Y != 0
    z = torch.as_tensor(st.sheet_z, device="cuda")[:, None, None]
    i = torch.arange(st.nx, device="cuda", dtype=torch.float64)[:, None] * d
    j = torch.arange(st.ny, device="cuda", dtype=torch.float64)[None, :] * d
    m = torch.zeros((len(x), 3), dtype=torch.complex128, device="cuda")
    m[:, 0] -= (z * d * Y).sum((1, 2, 3))
    m[:, 1] += (z * d * X).sum((1, 2, 3))
    m[:, 2] += (i * d * Y).sum((1, 2, 3)) - (j * d * X).sum((1, 2, 3))
    t, D = st.top, st.dense
    for p, (u, l) in enumerate(t.pair_layers):
        c = x[:, D.off_c + p * st.nx * st.ny: D.off_c + (p + 1) * st.nx * st.ny].reshape(len(x), st.nx, st.ny)
        dz = float(st.sheet_z[l] - st.sheet_z[u])
        m[:, 0] += (j * dz * c).sum((1, 2))
        m[:, 1] -= (i * dz * c).sum((1, 2))
    for b, br in enumerate(st.branches):
        ra, rb = st.pos(br.a), st.pos(br.b)
        m += x[:, D.off_b + b][:, None] * torch.as_tensor(np.cross(ra, rb), device="cuda")
    return kx / cx.clamp(min=1) / d, ky / cy.clamp(min=1) / d, (0.5 * m).cpu().numpy()


def _exact_psi(s):
    """The horizontal segments' vector potential along each strip: at its centre, or by a 3 x 3 Gauss rule over its cell
    when the centre lies within three pitches and two widths of the segment."""
    st, d = s["st"], s["st"].d
    idx = np.concatenate([np.c_[st.xa, np.zeros(len(st.xa), int)], np.c_[st.ya, np.ones(len(st.ya), int)]])
    idx = torch.as_tensor(idx, device="cuda")
    y_strip = idx[:, 3] == 1
    px = (idx[:, 1] + (~y_strip).double() / 2) * d
    py = (idx[:, 2] + y_strip.double() / 2) * d
    zk = torch.as_tensor(st.sheet_z, device="cuda")[idx[:, 0]]
    half = torch.as_tensor(st.sheet_t, device="cuda")[idx[:, 0]] / 2
    psi = torch.zeros(len(idx), dtype=torch.float64, device="cuda")
    node = [-0.5 * math.sqrt(0.6), 0.0, 0.5 * math.sqrt(0.6)]
    weight = [5 / 18, 8 / 18, 5 / 18]
    for seg in s["segments"]:
        a, b, width, cur = seg[0:3], seg[3:6], float(seg[6]), float(seg[7])
        if a[0] == b[0] and a[1] == b[1]:
            continue
        L = float(np.linalg.norm(b - a))
        u = (b - a) / L
        pz = torch.where(0.5 * (a[2] + b[2]) > zk, zk + half, zk - half)
        rmin = max(width / 2, 1e-7)

        def pot(qx, qy):
            dx, dy, dz = qx - a[0], qy - a[1], pz - a[2]
            pu = dx * u[0] + dy * u[1] + dz * u[2]
            rho = torch.sqrt((dx * dx + dy * dy + dz * dz - pu * pu).clamp(min=rmin * rmin))
            return 1e-7 * (torch.asinh((L - pu) / rho) + torch.asinh(pu / rho))

        t = (((px - a[0]) * u[0] + (py - a[1]) * u[1] + (pz - a[2]) * u[2]) / L).clamp(0, 1) * L
        dist = torch.sqrt((px - a[0] - t * u[0]) ** 2 + (py - a[1] - t * u[1]) ** 2 + (pz - a[2] - t * u[2]) ** 2)
        mean = sum(weight[m] * weight[n] * pot(px + node[m] * d, py + node[n] * d) for m in range(3) for n in range(3))
        A = torch.where(dist < 3 * d + 2 * width, mean, pot(px, py))
        psi += cur * torch.where(y_strip, float(u[1]), float(u[0])) * A
    return (d * psi).cpu().numpy()
