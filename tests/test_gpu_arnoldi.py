"""GPU: the three kernels of a Householder GMRES iteration (krylov.cu, k_gm_vec / k_gm_dot /
k_gm_orth) at the sizes where their split changes: CTAs of 32, 128 and 256 rows, systems just
below and above those limits, column tiles of eight and their remainders, more columns than the
rows of a block of the products over T (64), many partial sums (summed over groups of CTAs),
restarted cycles, complex double and float-float bases.

Against the oracle's gmres_custom on the same operator applications. FP64: the residual estimates
of every iteration agree within 1e-9 of the first one. Both run a backward-stable Householder
orthogonalisation (errors of some k sqrt(N) eps, below 1e-11 here) and the estimate is the norm of
a projected vector no longer than the first residual; the factor of 100 above it is left for the
operator's own condition. FP32: two runs whose vectors differ in their last bits round differently
in the operator, which is as good as another operator within its bound of 2e-5, so that bound
holds for the estimates too."""
import numpy as np
import pytest

from oracle import peec_oracle as O
from solver_gb300 import configs, frequency, mesher
from solver_gb300.operator import GpuOperator

pytestmark = pytest.mark.gpu


def _op(shape, p, freq):
    req = configs.random_mixed(shape, s=5e-5, p=p, seed=5, nports=1, freqs=[freq], tol=1e-8)
    out, freqs, _s, z0, grid = mesher.parse_request(req)
    esc, inc, cc, diag, exp, ports, le, _li, Zs = out
    op = GpuOperator(inc, exp, diag["P"])
    op.fill(cc["origin"], cc["sx"], cc["sy"], cc["sz"], esc["Lp"], esc["P"])
    fs = frequency.FrequencyState(2 * np.pi * freqs[0] * esc["freq"], esc, inc, diag, Zs, le, ports,
                                  z0)
    op.set_frequency(fs.w, fs.DZ, fs.Yle, fs.lu)
    return op


@pytest.mark.parametrize("shape,p,iters,restart,dtypes", [
    ((4, 3, 2), 1.0, 12, 0, (0, 1)), ((9, 9, 5), 0.6, 75, 0, (0, 1)), ((13, 12, 6), 0.7, 40, 0, (0,)),
    ((14, 12, 6), 0.75, 17, 8, (0, 1)), ((24, 20, 12), 0.45, 33, 0, (0, 1)),
    ((28, 24, 14), 0.6, 24, 9, (1,)), ((40, 32, 20), 0.6, 26, 0, (0, 1))], ids=str)
def test_estimates_match_the_oracle(shape, p, iters, restart, dtypes):
    op = _op(shape, p, 3e10)
    try:
        rng = np.random.default_rng(2)
        b = rng.standard_normal(op.N) + 1j * rng.standard_normal(op.N)
        kw = dict(restarted=True, restart=restart) if restart else {}
        outer = 2 if restart else iters
        inner = restart if restart else iters
        for prec in dtypes:
            x, flag, rel, it, rv = op.gmres(b, None, 1e-30, outer, precision=prec, **kw)
            xo, fo, ro, ito, rvo = O.gmres_custom(b, bool(restart), 1e-30, outer, None,
                                                  lambda v: op.matvec(v, prec),
                                                  restart=inner)
            m = min(len(rv), len(rvo))
            assert m >= min(inner, op.N) // 2, (len(rv), len(rvo))
            d = np.abs(np.asarray(rv)[:m] - np.asarray(rvo)[:m])
            assert np.max(d) <= (1e-9 if prec == 0 else 2e-5) * rvo[0], (prec, int(np.argmax(d)), float(np.max(d)) / rvo[0])
    finally:
        op.close()
