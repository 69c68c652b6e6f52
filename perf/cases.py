"""Timed cases of the solver path: what a program that uses this framework has it do.

Kinds of cases, each through a public entry point:

* ``apply``     one operator application y = M^-1 K x on device vectors
                (``GpuOperator.matvec_dev``): the inner product of every Krylov iteration, in
                FP32 (inner solves), float-float (refinement residuals) and FP64 (reference
                algorithm). The FP32 operator's result carries single precision and is handed
                on in single precision.
* ``gmres64``   one port solve of the reference algorithm (``port_rhs`` and ``gmres``) at an
                installed frequency.
* ``mixed``     one frequency point of one port in mixed precision: the frequency state
                formed on the device (``set_frequency_device``), ``port_rhs``, ``solve_mixed``.
* ``fill``      the nine generating rows of a geometry and their spectra
                (``GpuOperator.fill``), the rows returned.
* ``rcc``       two frequencies of a retarded sweep: the spectra and the frequency state of
                each, and an operator application.
* ``risfill``   the dense RIS blocks from the bodies' coordinates (``DenseOperator.fill``),
                read back as calcola_Lp / calcola_P return them.
* ``risapply``  one application of the dense RIS operator.

Geometries are those of ``solver_gb300.configs``: the crossbar, Bernoulli(0.3) grids of copper
and dielectric (the benchmark's), Bernoulli(0.25) copper grids (the batched sweep's).
"""
import math

import numpy as np
import torch

from solver_gb300 import configs, mesher, ris
from solver_gb300 import frequency as fq
from solver_gb300.operator import GpuOperator, row_dims

PREC = {"fp64": 0, "fp32": 1, "ff": 2}
EPS0 = 8.854187816997944e-12


def listed():
    return [
        # the smallest operator: the crossbar of the reference configuration, 528 unknowns;
        # launches and latency
        {"name": "apply32_crossbar", "kind": "apply", "geom": "crossbar", "nx": 20, "ny": 20,
         "nz": 4, "prec": "fp32"},
        # the largest grid of the batched frequency sweep
        {"name": "apply32_96x96x48", "kind": "apply", "geom": "copper", "nx": 96, "ny": 96,
         "nz": 48, "prec": "fp32"},
        # the benchmark's grid: the product every inner Krylov iteration makes
        {"name": "apply32_128x128x64", "kind": "apply", "geom": "mixed", "nx": 128, "ny": 128,
         "nz": 64, "prec": "fp32"},
        # the same grid's refinement residual
        {"name": "applyff_128x128x64", "kind": "apply", "geom": "mixed", "nx": 128, "ny": 128,
         "nz": 64, "prec": "ff"},
        # the reference algorithm's product at the odd extents of a 57x57x13 board
        {"name": "apply64_57x57x13", "kind": "apply", "geom": "mixed", "nx": 57, "ny": 57,
         "nz": 13, "prec": "fp64"},
        # the reference configuration itself: one port of the crossbar near 1 GHz to 1e-6
        {"name": "gmres64_crossbar", "kind": "gmres64", "geom": "crossbar", "nx": 20, "ny": 20,
         "nz": 4, "tol": 1e-6},
        # a middle grid of the batched sweep, one frequency point from a zero start
        {"name": "mixed_64x64x32", "kind": "mixed", "geom": "copper", "nx": 64, "ny": 64,
         "nz": 32, "warm": False},
        # a frequency point of the benchmark, started from its neighbour's solution
        {"name": "mixed_128x128x64", "kind": "mixed", "geom": "mixed", "nx": 128, "ny": 128,
         "nz": 64, "warm": True},
        # setting up the benchmark's geometry
        {"name": "fill_128x128x64", "kind": "fill", "nx": 128, "ny": 128, "nz": 64, "ay": 1.0,
         "az": 1.0},
        # two frequencies of a retarded sweep
        {"name": "rcc_48x48x24", "kind": "rcc", "nx": 48, "ny": 48, "nz": 24},
        # setting up a dense RIS problem from its bodies
        {"name": "risfill_24x24x8", "kind": "risfill", "nx": 24, "ny": 24, "nz": 8},
        # the dense operator of the benchmark's RIS mesh, inside the mixed solve
        {"name": "risapply32_40x40x16", "kind": "risapply", "nx": 40, "ny": 40, "nz": 16,
         "prec": "fp32"},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("apply", "apply", "apply", "gmres64", "mixed", "mixed", "fill", "rcc",
                       "risfill", "risapply"))
    if kind == "apply":
        return {"kind": kind, "geom": rng.choice(("copper", "mixed")), "nx": size(12, 128),
                "ny": size(12, 128), "nz": size(4, 64),
                "prec": rng.choice(("fp32", "fp32", "ff", "fp64"))}
    if kind == "gmres64":
        return {"kind": kind, "geom": rng.choice(("copper", "mixed")), "nx": size(12, 64),
                "ny": size(12, 64), "nz": size(4, 32), "tol": rng.choice((1e-6, 1e-8))}
    if kind == "mixed":
        return {"kind": kind, "geom": rng.choice(("copper", "mixed")), "nx": size(20, 128),
                "ny": size(20, 128), "nz": size(8, 64), "warm": rng.random() < 0.5}
    if kind == "fill":
        return {"kind": kind, "nx": size(12, 128), "ny": size(12, 128), "nz": size(4, 64),
                "ay": rng.choice((1.0, 1.0, 2.5, 5.0)), "az": rng.choice((1.0, 1.0, 0.5, 0.05))}
    if kind == "rcc":
        return {"kind": kind, "nx": size(16, 64), "ny": size(16, 64), "nz": size(6, 32)}
    if kind == "risfill":
        return {"kind": kind, "nx": size(8, 32), "ny": size(8, 32), "nz": size(4, 10)}
    return {"kind": kind, "nx": size(12, 40), "ny": size(12, 40), "nz": size(4, 16),
            "prec": rng.choice(("fp32", "fp32", "fp64"))}


# ------------------------------------------------------------------------------ inputs


def _mesh(case):
    """A geometry through the host mesher, as a solve request gives it. The occupancy goes by
    the case (configs' own seeds), vectors, frequencies and scalings by the seed."""
    shape = (case["nx"], case["ny"], case["nz"])
    geom = case.get("geom", "mixed")
    if geom == "crossbar":
        req = configs.crossbar_20x20x4()
    elif geom == "copper":
        req = configs.random_copper(shape, p=0.25)
    else:
        req = configs.random_mixed(shape, nports=1)
    out, _freqs, settings, z0, grid = mesher.parse_request(req)
    esc, inc, cc, diag, exp, ports, le, _li, Zs = out
    return {"esc": esc, "inc": inc, "cc": cc, "diag": diag, "exp": exp, "ports": ports, "le": le,
            "Zs": Zs, "z0": z0, "grid": grid, "settings": settings}


def _hz(seed, k=0):
    """A frequency of the sweep's upper decade, where the port currents are well determined."""
    return float(3e9 * (10 / 3) ** np.random.default_rng([seed, 77, k]).random())


def _state(g, hz, factor=True):
    w = 2 * math.pi * hz * g["esc"]["freq"]
    return fq.FrequencyState(w, g["esc"], g["inc"], g["diag"], g["Zs"], g["le"], g["ports"],
                             g["z0"], factor=factor)


def _operator(g, rcc=False):
    op = GpuOperator(g["inc"], g["exp"], g["diag"]["P"])
    cc, esc = g["cc"], g["esc"]
    fill = op.fill_rcc if rcc else op.fill
    fill(cc["origin"], cc["sx"], cc["sy"], cc["sz"], esc["Lp"], esc["P"])
    return op


def _vector(n, seed):
    r = np.random.default_rng([seed, 5])
    return r.standard_normal(n) + 1j * r.standard_normal(n)


def _device(v):
    x = torch.from_numpy(v).cuda()
    y = torch.empty_like(x)
    torch.cuda.synchronize()
    return x, y


def _cell(case, seed):
    """Cell edges of a fill: whole micrometres, as a user writes them."""
    s = 1e-6 * int(np.random.default_rng([seed, 9]).integers(20, 200))
    return s, s * case["ay"], s * case["az"]


def _ris(case):
    g = _mesh(case)
    cc = g["cc"]
    vol, sur = ris.voxel_bodies(g["inc"], g["exp"], g["grid"], (cc["sx"], cc["sy"], cc["sz"]))
    R = np.real(np.asarray(g["diag"]["R"])).sum(axis=1)
    Cd = np.real(np.asarray(g["diag"]["Cd"]))
    has = (Cd > 0).any(axis=1)
    eff = np.zeros(R.size)
    eff[has] = 1.0 / np.where(Cd[has] > 0, 1.0 / np.where(Cd[has] > 0, Cd[has], 1.0),
                              0.0).sum(axis=1)
    vol.update({"R": R, "Cd": eff, "indici_dielettrici": np.flatnonzero((R == 0) & (eff > 0)),
                "Zs_part": np.zeros(R.size)})
    return g, vol, sur


def _ris_state(g, vol, hz, diag_Lp, diag_P):
    return ris.RisState(2 * math.pi * hz * g["esc"]["freq"], g["esc"], g["inc"], diag_Lp, diag_P,
                        g["ports"], {}, vol, True, 50.0)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "fill":
        # the rows depend on the lattice only: two voxels are enough of an occupancy
        shape = (case["nx"], case["ny"], case["nz"])
        occ = np.zeros(shape, dtype=bool)
        occ[:2, 0, 0] = True
        cell = _cell(case, seed)
        req = configs.make_request({"copper": occ}, [dict(configs.COPPER)], cell,
                                   [((0, 0, 0), (1, 0, 0))], [1e9], 1e-8)
        out, _f, _s, _z, _grid = mesher.parse_request(req)
        esc, inc, cc, diag, exp = out[:5]
        op = GpuOperator(inc, exp, diag["P"])
        return {"op": op, "run": _run_fill, "cc": cc, "esc": esc}
    if kind == "risfill":
        g, vol, sur = _ris(case)
        scale = 0.5 + np.random.default_rng([seed, 3]).random()
        esc = dict(g["esc"], Lp=g["esc"]["Lp"] * scale, P=g["esc"]["P"] * scale)
        op = ris.DenseOperator.from_geometry(g["inc"], vol, sur, esc)
        return {"op": op, "run": _run_risfill, "vol": vol, "sur": sur, "esc": esc}
    if kind == "risapply":
        g, vol, sur = _ris(case)
        op = ris.DenseOperator.from_geometry(g["inc"], vol, sur, g["esc"])
        st = _ris_state(g, vol, _hz(seed), op.diag_Lp, op.diag_P)
        op.set_frequency(st.w, st.DZ, st.Yle, st.lu)
        x, y = _device(_vector(op.N, seed))
        return {"op": op, "run": _run_apply, "x": x, "y": y, "prec": PREC[case["prec"]]}
    g = _mesh(case)
    op = _operator(g, rcc=kind == "rcc")
    if kind == "apply":
        fs = _state(g, _hz(seed))
        op.set_frequency(fs.w, fs.DZ, fs.Yle, fs.lu)
        x, y = _device(_vector(op.N, seed))
        return {"op": op, "run": _run_apply, "x": x, "y": y, "prec": PREC[case["prec"]]}
    node = tuple(int(v) for v in np.asarray(g["ports"]["port_nodes"]).reshape(-1, 2)[0])
    if kind == "gmres64":
        hz = _hz(seed) if case["geom"] != "crossbar" else _hz(seed) / 4
        fs = _state(g, hz)
        op.set_frequency(fs.w, fs.DZ, fs.Yle, fs.lu)
        return {"op": op, "run": _run_gmres, "node": node, "Is": g["esc"]["Is"],
                "tol": case["tol"], "maxit": g["settings"]["Inner_Iter"]}
    # states formed on the device: the first frequency's host factors give their pattern
    hz0 = _hz(seed)
    fs = _state(g, hz0)
    op.set_frequency(fs.w, fs.DZ, fs.Yle, fs.lu)
    op.enable_refactor(fs.Yle)
    op.set_edge_state(g["diag"], g["Zs"], g["esc"])
    later = [_state(g, hz, factor=False) for hz in _later(seed)]
    if kind == "rcc":
        x, y = _device(_vector(op.N, seed))
        return {"op": op, "run": _run_rcc, "x": x, "y": y, "hz": _later(seed),
                "state": [(s.w, s.Yle) for s in later]}
    x0 = None
    if case["warm"]:
        b = op.port_rhs(*node, g["esc"]["Is"])
        x0 = op.solve_mixed(b, None, 1e-8)[0]
    return {"op": op, "run": _run_mixed, "node": node, "Is": g["esc"]["Is"], "x0": x0,
            "state": (later[0].w, later[0].Yle)}


def _later(seed):
    """The frequencies after the first: neighbours in a sweep."""
    return [_hz(seed) * 0.85, _hz(seed) * 0.72]


# ------------------------------------------------------------------------------ passes


def run(state):
    return state["run"](state)


def _result(y, prec):
    return y.to(torch.complex64) if prec == PREC["fp32"] else y


def _run_apply(s):
    s["op"].matvec_dev(s["x"].data_ptr(), s["y"].data_ptr(), s["prec"])
    return _result(s["y"], s["prec"])


def _run_gmres(s):
    op = s["op"]
    b = op.port_rhs(*s["node"], s["Is"])
    return op.gmres(b, None, s["tol"], s["maxit"])[0]


# the mixed solve's answer is asked for to 1e-10, two digits past the sweeps' threshold, as
# the port impedances of the accuracy studies are
MIXED_TOL = 1e-10


def _run_mixed(s):
    op = s["op"]
    op.set_frequency_device(*s["state"])
    b = op.port_rhs(*s["node"], s["Is"])
    return op.solve_mixed(b, s["x0"], MIXED_TOL)[0]


def _run_fill(s):
    cc, esc = s["cc"], s["esc"]
    return s["op"].fill(cc["origin"], cc["sx"], cc["sy"], cc["sz"], esc["Lp"], esc["P"],
                        return_rows=True)


def _run_rcc(s):
    op, out = s["op"], []
    for hz, state in zip(s["hz"], s["state"]):
        op.set_rcc_frequency(hz)
        op.set_frequency_device(*state)
        op.matvec_dev(s["x"].data_ptr(), s["y"].data_ptr(), PREC["fp32"])
        out.append(_result(s["y"], PREC["fp32"]))
    return out


def _run_risfill(s):
    s["op"].fill(s["vol"], s["sur"], s["esc"])
    Lp, P = s["op"].dense_data()
    return {**Lp, **P}


# ------------------------------------------------------------------------------ work


def _counts(case):
    """Edges, surfaces and nodes expected of the geometry."""
    cells = case["nx"] * case["ny"] * case["nz"]
    if case.get("geom") == "crossbar":
        return 272, 160, 96
    if case.get("geom") == "copper":
        return 0.18 * cells, 0.55 * cells, 0.22 * cells
    return 0.125 * cells, 0.415 * cells, 0.175 * cells


def _row_entries(case):
    return sum(int(np.prod(d)) for d in row_dims(case["nx"], case["ny"], case["nz"]).values())


def _conv_flops(case):
    """Six lattices, forward and inverse transforms at twice the extents, only the lines
    that hold or give something."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]

    def line(n):
        return 5 * 2 * n * math.log2(2 * n) if n > 1 else 0.0

    return 12 * (ny * nz * line(nx) + 2 * nx * nz * line(ny) + 4 * nx * ny * line(nz))


def _apply_work(case, item):
    """Vectors in and out, the generating rows in the arithmetic's width, topology, DZ, 1/P
    and the factors of SS (about four complex entries a node)."""
    m, ns, n = _counts(case)
    return (32 * (m + ns + n) + item * _row_entries(case) + 24 * m + 16 * ns + 80 * n,
            _conv_flops(case) + 40 * m + 12 * ns + 80 * n)


def work(case):
    kind = case["kind"]
    m, ns, n = _counts(case)
    N = m + ns + n
    if kind == "apply":
        b, f = _apply_work(case, {"fp32": 4, "ff": 8, "fp64": 8}[case["prec"]])
        return {"bytes": b, "flops": f}
    if kind in ("gmres64", "mixed"):
        its = 20  # iterations such a solve takes, each one application and its basis
        b, f = _apply_work(case, 8 if kind == "gmres64" else 4)
        return {"bytes": its * (b + 16 * N * its / 2), "flops": its * (f + 16 * N * its / 2)}
    if kind == "fill":
        e = _row_entries(case)
        return {"bytes": 8 * e, "flops": 400 * e}
    if kind == "rcc":
        b, f = _apply_work(case, 16)
        return {"bytes": 2 * b, "flops": 2 * (2 * f + _conv_flops(case))}
    pairs = (m / 3) ** 2 * 3 + ns ** 2
    if kind == "risfill":
        return {"bytes": 8 * pairs, "flops": 500 * pairs / 2}
    return {"bytes": (4 if case["prec"] == "fp32" else 8) * pairs + 32 * N, "flops": 4 * pairs}


# ------------------------------------------------------------------------------ 64 bits
# The same results in plain torch and numpy, complex128 / float64. The mesh, the generating
# rows, the dense blocks and the factors of SS are inputs of an application; the products,
# the solves and the integrals are computed here.

_ROW = (("p12_se", 0, 0, (1, 1, 1), (0, 0, 0)), ("p34_se", 1, 1, (1, 1, 1), (0, 0, 0)),
        ("p56_se", 2, 2, (1, 1, 1), (0, 0, 0)), ("p1234", 0, 1, (2, 2, 1), (1, -1, 0)),
        ("p1256", 0, 2, (1, 2, 2), (0, -1, 1)), ("p3456", 1, 2, (2, 1, 2), (-1, 0, 1)),
        ("Lpx", 3, 3, (1, 1, 1), (0, 0, 0)), ("Lpy", 4, 4, (1, 1, 1), (0, 0, 0)),
        ("Lpz", 5, 5, (1, 1, 1), (0, 0, 0)))


class _Conv:
    """LpI and PQ by one FFT product per block, from generating rows (float64 or complex)."""

    def __init__(self, g, rows):
        grid, inc, exp = g["grid"], g["inc"], g["exp"]
        d = row_dims(*grid)
        fam = [d["p12_se"], d["p34_se"], d["p56_se"], d["Lpx"], d["Lpy"], d["Lpz"]]
        self.L = [1 << (2 * n).bit_length() for n in (grid[2], grid[1], grid[0])]
        cut = np.cumsum([0] + [int(inc[k]) for k in ("mx", "my", "mz")])
        ec, sc = np.asarray(exp["edge_cell"]), np.asarray(exp["surf_cell"])
        sf = np.asarray(exp["surf_fam"])
        self.m, self.ns = int(cut[3]), sc.size
        at = [np.flatnonzero(sf == f) for f in range(3)]
        self.where = ([(self.m + a, sc[a]) for a in at] +
                      [(np.arange(cut[c], cut[c + 1]), ec[cut[c]:cut[c + 1]]) for c in range(3)])
        self.fam = fam
        self.blocks = []
        for key, fo, fi, s, o in _ROW:
            if key not in rows or not np.prod(fam[fo]) or not np.prod(fam[fi]):
                continue
            row = torch.as_tensor(np.asarray(rows[key])).cuda().reshape(d[key][::-1])
            self.blocks.append((fo, fi, self._spectrum(row, fam[fo], fam[fi], s, o)))
            if fo != fi:
                back = tuple(-v for v in o)
                self.blocks.append((fi, fo, self._spectrum(row, fam[fi], fam[fo], s, back)))

    def _spectrum(self, row, na, nb, s, o):
        k = row
        for dim, a in ((0, 2), (1, 1), (2, 0)):  # z, y, x
            L, M = self.L[dim], row.shape[dim]
            e = torch.arange(L)
            e = torch.where(e < na[a], e, e - L)
            t = (s[a] * e + o[a]).abs()
            ok = (e > -nb[a]) & (t < M)
            k = k.index_select(dim, t.clamp(max=M - 1).cuda())
            k = k * ok.cuda().to(k.dtype).reshape([-1 if q == dim else 1 for q in range(3)])
        return torch.fft.fftn(k.to(torch.complex128))

    def __call__(self, x):
        X = {}
        for f, (idx, cell) in enumerate(self.where):
            dims = self.fam[f]
            buf = np.zeros(int(np.prod(dims)), dtype=np.complex128)
            buf[cell] = x[idx]
            t = torch.from_numpy(buf.reshape(dims[::-1])).cuda()
            X[f] = torch.fft.fftn(t, s=self.L) if t.numel() else None
        out = np.zeros(self.m + self.ns, dtype=np.complex128)
        for f, (idx, cell) in enumerate(self.where):
            if X[f] is None or not idx.size:
                continue
            Y = sum(S * X[g] for fo, g, S in self.blocks if fo == f)
            d = self.fam[f]
            y = torch.fft.ifftn(Y)[:d[2], :d[1], :d[0]].reshape(-1).cpu().numpy()
            out[idx] = y[cell]
        return out[:self.m], out[self.m:]


def _exact_apply(inc, product, w, DZ, Yle, lu, invP, x):
    """y = M^-1 K x with the block preconditioner."""
    A, G = inc["A"], inc["Gamma"]
    m, ns = A.shape[0], G.shape[1]
    I, Q, Phi = x[:m], x[m:m + ns], x[m + ns:]
    LpI, PQ = product(x)
    Y1 = 1j * w * LpI + DZ * I + A @ Phi
    Y2 = PQ - G.T @ Phi
    Y3 = -(A.T @ I) + Yle @ Phi + 1j * w * (G @ Q)
    M = lu.solve(A.T @ (Y1 / DZ) - 1j * w * (G @ (invP * Y2)) + Y3)
    return np.concatenate([(Y1 - A @ M) / DZ, invP * (Y2 + G.T @ M), M])


def _exact_solve(apply, b, steps=70, tol=1e-13):
    """GMRES from zero, modified Gram-Schmidt twice over."""
    beta = np.linalg.norm(b)
    V, H = [b / beta], np.zeros((steps + 1, steps), dtype=np.complex128)
    for j in range(steps):
        v = apply(V[j])
        for _ in range(2):
            for i, u in enumerate(V):
                c = np.vdot(u, v)
                H[i, j] += c
                v = v - c * u
        H[j + 1, j] = np.linalg.norm(v)
        V.append(v / H[j + 1, j])
        e = np.zeros(j + 2, dtype=np.complex128)
        e[0] = beta
        y = np.linalg.lstsq(H[:j + 2, :j + 1], e, rcond=None)[0]
        if np.linalg.norm(H[:j + 2, :j + 1] @ y - e) <= tol * beta:
            break
    return sum(c * u for c, u in zip(y, V))


def _fin(t):
    return torch.nan_to_num(t, nan=0.0, posinf=0.0, neginf=0.0)


def _lg(t):
    return t.abs().log()


def _corners(n):
    return [tuple((c >> (n - 1 - k)) & 1 for k in range(n)) for c in range(1 << n)]


def _vol_vol(a, b):
    """Integral of 1/R over two bricks; a, b: per axis (low, high), broadcast together."""
    sol = 0.0
    for c in _corners(6):
        X, Y, Z = (a[k][c[k]] - b[k][c[3 + k]] for k in range(3))
        X2, Y2, Z2 = X * X, Y * Y, Z * Z
        R = (X2 + Y2 + Z2).sqrt()
        t = (X2 * X2 + Y2 * Y2 + Z2 * Z2 - 3 * X2 * Y2 - 3 * Y2 * Z2 - 3 * X2 * Z2) * R / 60
        for u, v, q, u2, v2 in ((Y, Z, X, Y2, Z2), (Y, X, Z, Y2, X2), (Z, X, Y, Z2, X2)):
            t = t + _fin((u2 * v2 / 4 - u2 * u2 / 24 - v2 * v2 / 24) * q * _lg(q + R))
            t = t - q.abs() * q * q * u * v / 6 * torch.atan2(u * v, q.abs() * R)
        sol = sol + (-1) ** (sum(c) + 1) * t
    return sol


def _para(ax, ay, z1, bx, by, z2):
    sol = 0.0
    for c in _corners(4):
        X, Y, Z = ax[c[0]] - bx[c[3]], ay[c[1]] - by[c[2]], z1 - z2
        R = (X * X + Y * Y + Z * Z).sqrt()
        t = (-1.0 / 6 * (X * X + Y * Y - 2 * Z * Z) * R -
             X * Y * Z.abs() * torch.atan2(X * Y, Z.abs() * R) +
             _fin(0.5 * (X * X - Z * Z) * Y * _lg(Y + R)) +
             _fin(0.5 * (Y * Y - Z * Z) * X * _lg(X + R)))
        sol = sol + (-1) ** sum(c) * t
    return sol


def _ortho(ax, ay, z1, bx, y2, bz):
    sol = 0.0
    for c in _corners(4):
        X, Y, Z = ax[c[0]] - bx[c[3]], ay[c[1]] - y2, z1 - bz[c[2]]
        R = (X * X + Y * Y + Z * Z).sqrt()
        t = (-1.0 / 3 * Y * Z * R - 0.5 * X * Z.abs() * Z * torch.atan2(X * Y, Z.abs() * R) -
             0.5 * X * Y.abs() * Y * torch.atan2(X * Z, Y.abs() * R) -
             1.0 / 6 * X.abs() * X * X * torch.atan2(Y * Z, X.abs() * R) +
             _fin(X * Y * Z * _lg(X + R)) + _fin((0.5 * X * X - Z * Z / 6) * Z * _lg(Y + R)) +
             _fin((0.5 * X * X - Y * Y / 6) * Y * _lg(Z + R)))
        sol = sol + (-1) ** sum(c) * t
    return sol


def _faces(p1, a, p2, b):
    """Integral over two faces with normals p1, p2; a, b: per axis (low, high, centre)."""
    if p1 == p2:
        u, v = [k for k in range(3) if k != p1]
        return _para(a[u], a[v], a[p1][2], b[u], b[v], b[p1][2])
    k = 3 - p1 - p2
    return _ortho(a[k], a[p2], a[p1][2], b[k], b[p2][2], b[p1])


def _exact_fill(case, seed):
    if case["ay"] != 1.0 or case["az"] != 1.0:
        return None  # flat or long cells: distant bodies take the collapsed closed forms
    s = _cell(case, seed)
    esc = {"Lp": 1e6, "P": 1e-12}
    dims = row_dims(case["nx"], case["ny"], case["nz"])

    def r14(t):
        return torch.round(t * 1e14) / 1e14

    def shaped(t, axis):
        return t.reshape([1, 1, -1] if axis == 0 else [1, -1, 1] if axis == 1 else [-1, 1, 1])

    out = {}
    for c, key in enumerate(("Lpx", "Lpy", "Lpz")):
        a, b = [], []
        for k in range(3):
            i = torch.arange(dims[key][k], dtype=torch.float64, device="cuda")
            lo = s[k] * i + s[k] / 2
            ctr = 0.5 * (lo + (s[k] * (i + 1) + s[k] / 2)) if k == c else lo
            t = [shaped(r14(ctr + q * s[k] / 2), k) for q in (-1, 1)]
            a.append([v.flatten()[0] for v in t])
            b.append(t)
        S = s[(c + 1) % 3] * s[(c + 2) % 3]
        row = (esc["Lp"] * 1e-7 / (S * S) * _vol_vol(a, b)).flatten()
        row[0] = 0.0
        out[key] = row
    normal = {1: (1, -1), 2: (1, 1), 3: (0, -1), 4: (0, 1), 5: (2, -1), 6: (2, 1)}
    for key, f1, f2 in (("p12_se", 1, 1), ("p34_se", 3, 3), ("p56_se", 5, 5), ("p1234", 3, 2),
                        ("p1256", 5, 2), ("p3456", 5, 4)):
        half = {"p1234": (1, 1, 0), "p1256": (0, 1, 1), "p3456": (1, 0, 1)}.get(key, (0, 0, 0))
        boxes = []
        for face in (f1, f2):
            p, side = normal[face]
            box = []
            for k in range(3):
                i = torch.arange(dims[key][k], device="cuda")
                ctr = s[k] * (i // 2 if half[k] else i).double() + s[k] / 2
                ctr = ctr + side * s[k] / 2 if k == p else ctr
                e = 0.0 if k == p else s[k]
                box.append([shaped(ctr + q * e / 2, k) for q in (-1, 1, 0)])
            boxes.append((p, box))
        (p1, a), (p2, b) = boxes
        a = [[v.flatten()[0] for v in t] for t in a]
        area = [np.prod([s[k] for k in range(3) if k != p]) for p in (p1, p2)]
        full = torch.zeros(dims[key][::-1], dtype=torch.float64, device="cuda")
        out[key] = (esc["P"] / (4 * math.pi * EPS0 * area[0] * area[1]) *
                    _faces(p1, a, p2, b) + full).flatten()
    return {k: v.cpu().numpy() for k, v in out.items()}


def _lp_self(length, W, T):
    """Self inductance of a bar, closed form."""
    w, t = W / length, T / length
    r, aw, at = np.sqrt(w * w + t * t), np.sqrt(w * w + 1), np.sqrt(t * t + 1)
    ar, ash = np.sqrt(w * w + t * t + 1), np.arcsinh
    g1 = 0.25 * (ash(w / at) / w + ash(t / aw) / t + ash(1 / r))
    g2 = (t * t / w * ash(w / (t * at * (r + ar))) + w * w / t * ash(t / (w * aw * (r + ar))) +
          t * t / (w * w) * ash(w * w / (t * r * (at + ar))) +
          w * w / (t * t) * ash(t * t / (w * r * (aw + ar))) +
          ash(w * t * t / (at * (aw + ar))) / (w * t * t) +
          ash(t * w * w / (aw * (at + ar))) / (t * w * w)) / 24
    g3 = (np.arctan(w * t / ar) / (w * t) + t / w * np.arctan(w / (t * ar)) +
          w / t * np.arctan(t / (w * ar))) / 6
    g4 = ((ar + r + t + at) * t * t / ((ar + r) * (r + t) * (t + at) * (at + ar)) +
          (ar + r + w + aw) * w * w / ((ar + r) * (r + w) * (w + aw) * (aw + ar)) +
          (ar + aw + 1 + at) / ((ar + aw) * (aw + 1) * (1 + at) * (at + ar))) / 60
    g5 = (1 / (r + ar) + 1 / (aw + ar) + 1 / (at + ar)) / 20
    return 2 * 4e-7 * length * (g1 + g2 - g3 - g4 - g5)


def _exact_risfill(case, seed):
    g, vol, sur = _ris(case)
    scale = 0.5 + np.random.default_rng([seed, 3]).random()
    esc = {k: g["esc"][k] * scale for k in ("Lp", "P")}
    cut = np.cumsum([0] + [int(g["inc"][k]) for k in ("mx", "my", "mz")])
    v = np.asarray(vol["coordinate"]).reshape(-1, 8, 3)
    out = {}

    def sides(lo, hi, col):
        lo, hi = np.round(lo, 14), np.round(hi, 14)
        t = [(a, b, 0.5 * (a + b)) for a, b in zip(lo.T, hi.T)]
        shape = (1, -1) if col else (-1, 1)
        return [[torch.as_tensor(np.ascontiguousarray(q)).cuda().reshape(shape) for q in k]
                for k in t]

    def upper(full):
        """Pairs are integrated once, row body first: the lower triangle mirrors."""
        u = torch.triu(full)
        return (u + torch.triu(full, 1).T).cpu().numpy()

    for c, key in enumerate(("Lp_x", "Lp_y", "Lp_z")):
        b = v[cut[c]:cut[c + 1]]
        lo, hi = b.min(axis=1), b.max(axis=1)
        S = torch.as_tensor(np.asarray(vol["S"])[cut[c]:cut[c + 1]]).cuda()
        full = upper(1e-7 / (S[:, None] * S[None, :]) *
                     _vol_vol(sides(lo, hi, False), sides(lo, hi, True)) * esc["Lp"])
        d = hi - lo
        np.fill_diagonal(full, _lp_self(d[:, c], d[:, (c + 1) % 3], d[:, (c + 2) % 3]) * esc["Lp"])
        out[key] = full
    e = np.asarray(sur["estremi_celle"])
    lo, hi = np.minimum(e[:, :3], e[:, 9:]), np.maximum(e[:, :3], e[:, 9:])
    nrm = np.argmin(np.round(hi, 14) - np.round(lo, 14), axis=1)
    S = torch.as_tensor(np.asarray(sur["S"])).cuda()
    P = torch.zeros((S.numel(), S.numel()), dtype=torch.float64, device="cuda")
    for p1 in range(3):
        r = np.flatnonzero(nrm == p1)
        for p2 in range(3):
            q = np.flatnonzero(nrm == p2)
            val = _faces(p1, sides(lo[r], hi[r], False), p2, sides(lo[q], hi[q], True))
            P[torch.as_tensor(r).cuda()[:, None], torch.as_tensor(q).cuda()[None, :]] = val
    out["P"] = upper(P / (4 * math.pi * EPS0 * S[:, None] * S[None, :]) * esc["P"])
    return out


def _rcc_rows(g, rows, hz):
    """The rows times exp(-j beta R), R the distance of the generating cell."""
    cc, grid = g["cc"], g["grid"]
    s = (cc["sx"], cc["sy"], cc["sz"])
    beta = 2 * math.pi * hz * math.sqrt(EPS0 * 4e-7 * math.pi)
    shift = {"p1234": ((0, -1), (1, 1), (1, 1, 0)), "p1256": ((2, -1), (1, 1), (0, 1, 1)),
             "p3456": ((2, -1), (0, 1), (1, 0, 1))}
    out = {}
    for key, d in row_dims(*grid).items():
        if key not in rows or not np.prod(d):
            continue
        (p1, s1), (p2, s2), half = shift.get(key, ((0, 0), (0, 0), (0, 0, 0)))
        r2 = 0.0
        for k in range(3):
            i = np.arange(d[k])
            t = s[k] * (i // 2 if half[k] else i).astype(np.float64)
            t = t + (s2 * s[k] / 2 if k == p2 else 0.0) - (s1 * s[k] / 2 if k == p1 else 0.0)
            r2 = r2 + (t * t).reshape([-1 if q == 2 - k else 1 for q in range(3)])
        out[key] = np.asarray(rows[key]).reshape(d[::-1]) * np.exp(-1j * beta * np.sqrt(r2))
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "fill":
        return _exact_fill(case, seed)
    if kind == "risfill":
        return _exact_risfill(case, seed)
    if kind == "risapply":
        g, vol, sur = _ris(case)
        op = ris.DenseOperator.from_geometry(g["inc"], vol, sur, g["esc"])
        Lp, P = op.dense_data()
        st = _ris_state(g, vol, _hz(seed), op.diag_Lp, op.diag_P)
        x, invP = _vector(op.N, seed), 1.0 / op.diag_P
        op.close()
        cut = np.cumsum([0] + [int(g["inc"][k]) for k in ("mx", "my", "mz")])

        def dense(M, v):
            t = torch.from_numpy(v).cuda()
            Md = torch.from_numpy(np.ascontiguousarray(M)).cuda()
            return torch.complex(Md @ t.real, Md @ t.imag).cpu().numpy()

        def product(x):
            I = x[:cut[3]]
            LpI = [dense(M, I[a:b]) - np.diag(M) * I[a:b] for M, a, b in
                   ((Lp[k], cut[c], cut[c + 1]) for c, k in enumerate(("Lp_x", "Lp_y", "Lp_z")))]
            return np.concatenate(LpI), dense(P["P"], x[cut[3]:cut[3] + invP.size])

        return _exact_apply(g["inc"], product, st.w, st.DZ, st.Yle, st.lu, invP, x)
    g = _mesh(case)
    invP = 1.0 / np.asarray(g["diag"]["P"]).ravel()
    op = GpuOperator(g["inc"], g["exp"], g["diag"]["P"])
    cc, esc = g["cc"], g["esc"]
    args = (cc["origin"], cc["sx"], cc["sy"], cc["sz"], esc["Lp"], esc["P"])
    rows = op.fill_rcc(*args) if kind == "rcc" else op.fill(*args, return_rows=True)
    N = op.N
    op.close()

    def applied(product, fs, x):
        return _exact_apply(g["inc"], product, fs.w, fs.DZ, fs.Yle, fs.lu, invP, x)

    if kind == "rcc":
        return [applied(_Conv(g, _rcc_rows(g, rows, hz)), _state(g, hz), _vector(N, seed))
                for hz in _later(seed)]
    product = _Conv(g, rows)
    if kind == "apply":
        return applied(product, _state(g, _hz(seed)), _vector(N, seed))
    if kind == "mixed":
        hz = _later(seed)[0]
    else:
        hz = _hz(seed) if case["geom"] != "crossbar" else _hz(seed) / 4
    fs = _state(g, hz)
    m, ns = g["inc"]["A"].shape[0], g["inc"]["Gamma"].shape[1]
    n1, n2 = np.asarray(g["ports"]["port_nodes"]).reshape(-1, 2)[0]
    rhs = np.zeros(N - m - ns, dtype=np.complex128)
    rhs[n1] += esc["Is"]
    rhs[n2] -= esc["Is"]
    M = fs.lu.solve(rhs)  # M^-1 [0; 0; rhs]
    b = np.concatenate([-(g["inc"]["A"] @ M) / fs.DZ, invP * (g["inc"]["Gamma"].T @ M), M])
    return _exact_solve(lambda v: applied(product, fs, v), b)
