"""GPU: the groups' solves that form their own node sums (sparse.cu, k_sptrsv_grp with NODE), with
a general diagonal of L and with a row scaling (peec_set_frequency's row_scale, for factors of
scaled rows such as UMFPACK's): the operator does not depend on how SS was factorised. Bound: two
factorisations of one SS agree to 1e-10 (the parity tests' bound), or 20 times the operator's
response to inputs changed in the last bit."""
import numpy as np
import pytest
import scipy.sparse as sp
from scipy.sparse.linalg import splu

from solver_gb300 import _lib, configs, frequency, mesher
from solver_gb300.operator import GpuOperator

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def system():
    req = configs.random_mixed((12, 11, 6), s=5e-5, p=0.5, seed=9, nports=2, freqs=[2e9], tol=1e-8)
    out, freqs, _s, z0, _grid = mesher.parse_request(req)
    esc, inc, cc, diag, exp, ports, le, _li, Zs = out
    op = GpuOperator(inc, exp, diag["P"])
    op.fill(cc["origin"], cc["sx"], cc["sy"], cc["sz"], esc["Lp"], esc["P"])
    fs = frequency.FrequencyState(2 * np.pi * freqs[0] * esc["freq"], esc, inc, diag, Zs, le, ports,
                                  z0)
    A, G = inc["A"], inc["Gamma"]
    SS = (A.T @ sp.diags(1 / np.asarray(fs.DZ).ravel()) @ A +
          1j * fs.w * (G @ sp.diags(1 / np.asarray(diag["P"]).ravel()) @ G.T) + fs.Yle).tocsc()
    yield op, fs, SS
    op.close()


def _install(op, fs, L, U, pr, pc, rs):
    """peec_set_frequency with given factors and row scaling"""
    def csr(M):
        M = M.tocsr()
        M.sort_indices()
        return (M.indptr.astype(np.int64), M.indices.astype(np.int64),
                np.ascontiguousarray(M.data.astype(np.complex128)).view(np.float64))

    (Lp, Lc, Lv), (Up, Uc, Uv) = csr(L), csr(U)
    Y = sp.coo_matrix(fs.Yle)
    yr, yc = Y.row.astype(np.int64), Y.col.astype(np.int64)
    yv = np.ascontiguousarray(Y.data.astype(np.complex128)).view(np.float64)
    DZ = np.ascontiguousarray(np.asarray(fs.DZ, dtype=np.complex128).ravel()).view(np.float64)
    pr, pc = pr.astype(np.int64), pc.astype(np.int64)
    p = _lib.ptr
    _lib.check(op.h, op.L.peec_set_frequency(
        op.h, fs.w, p(DZ), int(yr.size), p(yr), p(yc), p(yv), p(Lp), p(Lc), p(Lv), p(Up), p(Uc), p(Uv),
        p(pr), p(pc), None if rs is None else p(rs)))


@pytest.mark.parametrize("general_l", [False, True])
@pytest.mark.parametrize("scaled", [False, True])
@pytest.mark.parametrize("limit", [512, 4])
def test_factor_forms(system, general_l, scaled, limit):
    op, fs, SS = system
    rng = np.random.default_rng(4)
    n = op.n
    x = rng.standard_normal(op.N) + 1j * rng.standard_normal(op.N)
    op.set_lu_component_max(512)
    op.set_frequency(fs.w, fs.DZ, fs.Yle, fs.lu)
    ref = op.matvec(x, 0)
    peak, eps = np.max(np.abs(ref)), np.finfo(float).eps
    noise = np.max(np.abs(op.matvec(x * (1 + eps * rng.choice([-1, 1], op.N)), 0) - ref))
    rs = np.ascontiguousarray(0.5 + rng.random(n)) if scaled else None
    lu = splu((sp.diags(rs) @ SS if scaled else SS).tocsc(), permc_spec="MMD_AT_PLUS_A",
              options={"Equil": False})
    L, U = lu.L, lu.U
    if general_l:
        d = (0.7 + 0.6 * rng.random(n)) * np.exp(1j * rng.random(n))
        L, U = L @ sp.diags(d), sp.diags(1 / d) @ U
    op.set_lu_component_max(limit)  # 4: rows left for the global scheme, node sums in their own kernel
    _install(op, fs, L, U, lu.perm_r, lu.perm_c, rs)
    try:
        got = op.matvec(x, 0)
        assert np.max(np.abs(got - ref)) <= max(1e-10 * peak, 20 * noise)
        port = op.port_rhs(0, n - 1, 1.0)
        op.set_lu_component_max(512)
        op.set_frequency(fs.w, fs.DZ, fs.Yle, fs.lu)
        want = op.port_rhs(0, n - 1, 1.0)
        assert np.max(np.abs(port - want)) <= 1e-9 * np.max(np.abs(want))
    finally:
        op.set_lu_component_max(512)
