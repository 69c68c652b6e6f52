"""GPU: the LU solves by groups of components (sparse.cu, k_sptrsv_grp) at the sizes where
the packing and the lanes per row change: single rows, components around a warp, around the
packing limit, around the largest component a CTA takes and above it (the global scheme);
short and long rows, unit and general diagonals of L, row scaling by the permutations.

The solve is checked by its componentwise backward error. Each of the two triangular solves
forms a row's sum of k products in some order and divides by (multiplies with the inverse
of) the diagonal, so the computed x satisfies |LU x - b| <= c eps (|L||U||x| + |b|) with
c = 2 (k + 8): k additions and as many complex products (three roundings each) in each of
the two triangles."""
import numpy as np
import pytest
import scipy.sparse as sp

from solver_gb300 import ris
from solver_gb300.frequency import ExportedLU

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _factors(sizes, kmax, unit, seed):
    """Block-diagonal L and U (complex, well conditioned) with the given component sizes and
    up to kmax off-diagonal entries a row, each row linked to its component's previous row."""
    rng = np.random.default_rng(seed)
    rows, cols = [], []
    at = 0
    for s in sizes:
        for r in range(1, s):
            k = min(r, 1 + int(rng.integers(0, kmax)))
            c = np.unique(np.append(rng.choice(r, size=k, replace=False), r - 1))[-k:]
            rows += [at + r] * c.size
            cols += list(at + c)
        at += s
    n = at

    def values(m):
        return rng.standard_normal(m) + 1j * rng.standard_normal(m)

    off = 0.5 / kmax
    L = sp.coo_matrix((off * values(len(rows)), (rows, cols)), shape=(n, n))
    U = sp.coo_matrix((off * values(len(rows)), (cols, rows)), shape=(n, n))
    dl = np.ones(n) if unit else 1.0 + 0.3 * values(n) / 3
    du = 1.5 + 0.3 * values(n) / 3
    return (L + sp.diags(dl)).tocsr(), (U + sp.diags(du)).tocsr()


def _csr(M):
    M.sort_indices()
    return (M.indptr.astype(np.int64), M.indices.astype(np.int64),
            np.ascontiguousarray(M.data.astype(np.complex128)).view(np.float64))


@pytest.mark.parametrize("sizes,kmax,unit", [
    ([2], 1, True), ([1] * 37 + [2, 3], 1, True), ([31, 32, 33], 5, True),
    ([63, 64, 65, 1, 1], 9, False), ([255, 256, 257], 3, True), ([511, 512], 18, False),
    ([513, 40, 7], 6, True), ([20] * 700 + [1] * 900, 4, True), ([9] * 3000, 2, False),
    ([512, 300, 64, 64, 5, 5, 5], 30, True)])
def test_group_solves(sizes, kmax, unit):
    n = int(np.sum(sizes))
    L, U = _factors(sizes, kmax, unit, seed=n + kmax)
    rng = np.random.default_rng(n)
    pr, pc = rng.permutation(n), rng.permutation(n)
    inc = {"mx": 1, "my": 0, "mz": 0,
           "A": sp.csr_matrix(([-1.0, 1.0], ([0, 0], [0, n - 1])), shape=(1, n)),
           "Gamma": sp.csc_matrix(([1.0], ([0], [0])), shape=(n, 1))}
    Z = np.zeros((0, 0))
    op = ris.DenseOperator(inc, {"Lp_x": np.ones((1, 1)), "Lp_y": Z, "Lp_z": Z},
                           {"P": np.ones((1, 1))})
    try:
        op.set_frequency(1.0, np.ones(1, dtype=complex), sp.csr_matrix((n, n), dtype=complex),
                         ExportedLU((_csr(L), _csr(U), pr, pc)))
        n1, n2 = 0, n // 2 if n > 2 else 1
        x = op.port_rhs(n1, n2, 3.0)[2:]
    finally:
        op.close()
    b = np.zeros(n, dtype=complex)
    b[n1], b[n2] = 3.0, -3.0
    bp = np.empty(n, dtype=complex)
    bp[pr] = b  # Pr b
    z = np.empty(n, dtype=complex)
    z[pc] = x  # x = Pc z
    resid = np.abs(L @ (U @ z) - bp)
    scale = abs(L) @ (abs(U) @ np.abs(z)) + np.abs(bp)
    assert np.all(np.isfinite(x))
    # the residual itself is formed in doubles: as many roundings again
    assert np.all(resid <= 4 * (kmax + 8) * EPS * scale), float(np.max(resid / scale))
