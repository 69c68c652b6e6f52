"""GPU: a frequency state that could not be installed is not used. peec_set_frequency replaces
the context's arrays one by one, and the LU groups' plan holds positions in the ones before, so a
refused upload has to leave a context that refuses applications and solves (PEEC_ERR_STATE, by the
host's check, before anything is launched) until a whole state is installed; what then comes out is
what came out before, bit for bit (the same kernels on the same values)."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp
from scipy.sparse.linalg import splu

from solver_gb300 import _lib, configs, frequency, mesher
from solver_gb300.operator import GpuOperator

pytestmark = pytest.mark.gpu

OOM, BADARG, STATE = -2, -5, -7  # PEEC_ERR_*


def _geometry():
    req = configs.random_mixed((9, 8, 5), s=5e-5, p=0.6, seed=5, nports=1, freqs=[1e9], tol=1e-8)
    out, freqs, _s, z0, _grid = mesher.parse_request(req)
    esc, inc, cc, diag, exp, ports, le, _li, Zs = out
    fs = frequency.FrequencyState(2 * np.pi * freqs[0] * esc["freq"], esc, inc, diag, Zs, le, ports,
                                  z0)
    op = GpuOperator(inc, exp, diag["P"])
    op.fill(cc["origin"], cc["sx"], cc["sy"], cc["sz"], esc["Lp"], esc["P"])
    return op, fs, (diag, Zs, esc)


@pytest.fixture(scope="module")
def geom():
    op, fs, _data = _geometry()
    yield op, fs
    op.close()


def _refused(op, fs, fault):
    """set_frequency with an empty Yle and one fault; the code it returns"""
    (Lp, Lc, Lv), (Up, Uc, Uv), pr, pc = [
        tuple(np.array(v) for v in t) if isinstance(t, tuple) else np.array(t)
        for t in frequency.export_lu(fs.lu)]
    yr, yc, yv = np.zeros(1, np.int64), np.zeros(1, np.int64), np.zeros(2)
    nnz = 0
    r = op.n // 2
    if fault == "yle":
        nnz, yr[0] = 1, op.n
    elif fault == "permutation":
        pc[r] = op.n
    elif fault == "pivot":
        at = Up[r] + int(np.flatnonzero(Uc[Up[r]:Up[r + 1]] == r)[0])
        Uv[2 * at:2 * at + 2] = 0.0
    elif fault == "side":
        Lc[Lp[0]] = op.n - 1
    DZ = np.ascontiguousarray(np.asarray(fs.DZ, dtype=np.complex128).ravel())
    p = _lib.ptr
    return op.L.peec_set_frequency(op.h, fs.w, p(DZ.view(np.float64)), nnz, p(yr), p(yc), p(yv), p(Lp),
                                   p(Lc), p(Lv), p(Up), p(Uc), p(Uv), p(pr), p(pc), None)


def _is_refused(call):
    with pytest.raises(_lib.PeecError) as e:
        call()
    assert e.value.code == STATE


@pytest.mark.parametrize("fault", ["yle", "permutation", "pivot", "side"])
def test_refused_frequency_is_not_used(geom, fault):
    op, fs = geom
    rng = np.random.default_rng(1)
    x = rng.standard_normal(op.N) + 1j * rng.standard_normal(op.N)
    op.set_frequency(fs.w, fs.DZ, fs.Yle, fs.lu)
    op.enable_refactor(fs.Yle)
    y = op.matvec(x, 0)
    assert sp.coo_matrix(fs.Yle).nnz > 0
    assert _refused(op, fs, fault) == BADARG
    for call in (lambda: op.matvec(x, 0), lambda: op.matvec(x, 1), lambda: op.port_rhs(0, 1, 1.0),
                 lambda: op.gmres(x, None, 1e-6, 5), lambda: op.solve_mixed(x, None, 1e-6),
                 lambda: op.enable_refactor(fs.Yle)):
        _is_refused(call)
    op.set_lu_component_max(512)  # no plan is built for factors that are not there
    _is_refused(lambda: op.matvec(x, 0))
    if fault in ("yle", "permutation"):  # refused before anything was replaced: the plan stands
        op.set_frequency_refactor(fs.w, fs.DZ, fs.Yle)
        assert np.array_equal(op.matvec(x, 0), y)
    else:
        _is_refused(lambda: op.set_frequency_refactor(fs.w, fs.DZ, fs.Yle))
    op.set_frequency(fs.w, fs.DZ, fs.Yle, fs.lu)
    op.enable_refactor(fs.Yle)
    assert np.array_equal(op.matvec(x, 0), y)


def test_new_plan_keeps_the_state(geom):
    """Another component limit rebuilds the plan: the frequency state and the refactorisation
    plan stay installed. The rows of the global scheme sum in another order than the groups:
    the operator's bound of 1e-10, and 20 times its response to inputs changed in the last bit."""
    op, fs = geom
    rng = np.random.default_rng(2)
    x = rng.standard_normal(op.N) + 1j * rng.standard_normal(op.N)
    op.set_frequency(fs.w, fs.DZ, fs.Yle, fs.lu)
    op.enable_refactor(fs.Yle)
    y = op.matvec(x, 0)
    peak = np.max(np.abs(y))
    eps = np.finfo(float).eps
    noise = np.max(np.abs(op.matvec(x * (1 + eps * rng.choice([-1, 1], op.N)), 0) - y))
    bound = max(1e-10 * peak, 20 * noise)
    try:
        for limit in (0, 8):
            op.set_lu_component_max(limit)
            assert np.max(np.abs(op.matvec(x, 0) - y)) <= bound
            op.set_frequency_refactor(fs.w, fs.DZ, fs.Yle)
            assert np.max(np.abs(op.matvec(x, 0) - y)) <= bound
    finally:
        op.set_lu_component_max(512)
    assert np.array_equal(op.matvec(x, 0), y)


def test_wider_yle_pattern_at_the_set_up(geom):
    """enable_refactor with a pattern that has an admittance more than the installed Yle: the
    operator does not change by its zero, and a later frequency with that admittance is the one
    that host factors of the same SS give. Bounds: two factorisations of one SS agree to 1e-10 (as
    in test_gpu_refactor) or 20 times the operator's response to inputs changed in the last bit. A
    pattern without the installed admittances is refused and changes nothing."""
    op, fs = geom
    rng = np.random.default_rng(3)
    x = rng.standard_normal(op.N) + 1j * rng.standard_normal(op.N)
    op.set_frequency(fs.w, fs.DZ, fs.Yle, fs.lu)
    y = op.matvec(x, 0)
    peak, eps = np.max(np.abs(y)), np.finfo(float).eps
    noise = np.max(np.abs(op.matvec(x * (1 + eps * rng.choice([-1, 1], op.N)), 0) - y))
    bound = max(1e-10 * peak, 20 * noise)
    with pytest.raises(_lib.PeecError) as e:
        op.enable_refactor(sp.csr_matrix((op.n, op.n), dtype=complex))
    assert e.value.code == BADARG
    assert np.array_equal(op.matvec(x, 0), y)
    a, b = 1, op.n - 2
    g = 0.02 + 0.01j
    wide = (sp.csr_matrix(fs.Yle) +
            sp.csr_matrix(([g, g, -g, -g], ([a, b, a, b], [a, b, b, a])), shape=(op.n, op.n))).tocsr()
    assert wide.nnz > sp.coo_matrix(fs.Yle).nnz
    op.enable_refactor(wide)
    assert np.max(np.abs(op.matvec(x, 0) - y)) <= bound
    op.set_frequency_refactor(fs.w, fs.DZ, wide)
    got = op.matvec(x, 0)
    inc, _exp, diagP = op._init_args[:3]
    A, G = inc["A"], inc["Gamma"]
    SS = (A.T @ sp.diags(1 / np.asarray(fs.DZ).ravel()) @ A +
          1j * fs.w * (G @ sp.diags(1 / np.asarray(diagP).ravel()) @ G.T) + wide)
    op.set_frequency(fs.w, fs.DZ, wide, splu(sp.csc_matrix(SS), options={"Equil": False}))
    ref = op.matvec(x, 0)
    assert np.max(np.abs(got - ref)) <= max(bound, 1e-10 * np.max(np.abs(ref)))
    assert np.max(np.abs(ref - y)) > 10 * bound  # the admittance is seen


@pytest.mark.parametrize("valid", [False, True])
def test_new_topology_drops_what_was_installed(valid):
    """A second topology on a context, refused or not: nothing of the first one is used with it
    (its factors, refactorisation plan and edge data have other sizes)."""
    op, fs, data = _geometry()
    try:
        x = np.ones(op.N, dtype=complex)
        op.set_frequency(fs.w, fs.DZ, fs.Yle, fs.lu)
        op.enable_refactor(fs.Yle)
        op.set_edge_state(data[0], data[1], data[2])
        op.matvec(x, 0)
        n1, n2 = np.zeros(op.m, np.int64), np.ones(op.m, np.int64)
        n2[-1] = 1 if valid else op.n
        node = np.zeros(op.ns, np.int64)
        rc = op.L.peec_set_incidence(op.h, op.m, 0, 0, _lib.ptr(n1), _lib.ptr(n2), op.ns,
                                     _lib.ptr(node), op.n)
        assert rc == (0 if valid else BADARG)
        for call in (lambda: op.matvec(x, 0), lambda: op.port_rhs(0, 1, 1.0),
                     lambda: op.gmres(x, None, 1e-6, 5), lambda: op.solve_mixed(x, None, 1e-6),
                     lambda: op.set_frequency_refactor(fs.w, fs.DZ, fs.Yle),
                     lambda: op.set_frequency_device(fs.w, fs.Yle),
                     lambda: op.enable_refactor(fs.Yle)):
            _is_refused(call)
    finally:
        op.close()


def test_refused_allocation_leaves_the_context_usable():
    """An allocation the device refuses (a reduction scratch of 5 TB, at once) is reported as such
    and not a second time by the next call's launch checks; the scratch a fill leaves mapped (here
    some 33 MB of rows and transforms) is free again for others by then, and the next fill maps it
    once more, with the same rows."""
    import torch
    req = configs.random_mixed((48, 48, 24), s=5e-5, p=0.02, seed=5, nports=1, freqs=[1e9], tol=1e-8)
    out = mesher.parse_request(req)[0]
    esc, inc, cc, diag, exp = out[:5]
    op = GpuOperator(inc, exp, diag["P"])
    try:
        args = (cc["origin"], cc["sx"], cc["sy"], cc["sz"], esc["Lp"], esc["P"])
        rows = op.fill(*args, return_rows=True)
        v = torch.zeros(16, dtype=torch.complex128, device="cuda")
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        p = ctypes.c_void_p(v.data_ptr())
        assert op.L.peec_multidot(op.h, p, 10**6, p, 10**6, 1 << 30, p) == OOM
        assert torch.cuda.mem_get_info()[0] >= free + (16 << 20)
        again = op.fill(*args, return_rows=True)
        assert all(np.array_equal(rows[k], again[k]) for k in rows)
    finally:
        op.close()
