"""GPU: Arnoldi cycles of more columns than the last CTA's shared memory takes (krylov.cu: from 384
columns on k_gm_orth's sums and rotations, from 1,537 on k_gm_dot's sums are in global memory) and
a solution update from more coefficients than 48 KB hold (from 1,537 on).

Random signs on the generating rows leave an operator that hardly converges, so that long cycles
are run to their end. The last estimate is compared with the residual of the solution: a
backward-stable Householder solve solves a problem perturbed by some k 2^-53 |A| |x| (|A| as its
Frobenius norm, sqrt(N) times the mean gain of random vectors). That has to be below 1e-3 of the
right-hand side to say something: a wrong column of R or of the basis moves the estimate or the
solution by more."""
import numpy as np
import pytest

from solver_gb300 import configs, frequency, mesher
from solver_gb300.operator import GpuOperator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,iters", [((9, 9, 5), 420), ((17, 16, 9), 1600)], ids=str)
def test_long_cycle(shape, iters):
    req = configs.random_mixed(shape, s=5e-5, p=0.6, seed=5, nports=1, freqs=[3e10], tol=1e-8)
    out, freqs, _s, z0, _grid = mesher.parse_request(req)
    esc, inc, cc, diag, exp, ports, le, _li, Zs = out
    op = GpuOperator(inc, exp, diag["P"])
    try:
        rows = op.fill(cc["origin"], cc["sx"], cc["sy"], cc["sz"], esc["Lp"], esc["P"],
                       return_rows=True)
        rng = np.random.default_rng(6)
        op.set_rows({k: v * rng.choice([-1, 1], v.size) for k, v in rows.items()})
        fs = frequency.FrequencyState(2 * np.pi * freqs[0] * esc["freq"], esc, inc, diag, Zs, le,
                                      ports, z0)
        op.set_frequency(fs.w, fs.DZ, fs.Yle, fs.lu)
        assert op.N > iters + 50
        v = rng.standard_normal((8, op.N)) + 1j * rng.standard_normal((8, op.N))
        gain = np.sqrt(np.mean([np.linalg.norm(op.matvec(u, 0)) ** 2 / np.linalg.norm(u) ** 2
                                for u in v]))
        b = v[0]
        x, _flag, _rel, _it, rv = op.gmres(b, None, 1e-30, iters, precision=0)
        assert len(rv) == iters + 1, len(rv)
        true = np.linalg.norm(b - op.matvec(x, 0))
        bound = 4 * iters * 2.0**-53 * (np.sqrt(op.N) * gain * np.linalg.norm(x) +
                                        np.linalg.norm(b))
        assert bound < 1e-3 * rv[0], (bound, rv[0])
        assert abs(true - rv[-1]) <= bound, (true, rv[-1], bound)
    finally:
        op.close()
