"""GPU: the pair x and y passes (fftconv_impl.cuh, k_xpair and k_ypair) at every circulant length
they take along x and y (2 to 512 points, where the split of a line over threads changes),
with every entry of the half occupied or few of them, lines that
do not fill a CTA, ragged extents of the other axes and absent edge families.

The FP32 and the float-float operator against the FP64 one, whose passes are the direct kernels:
2e-5 and 1e-11 relative (max-norm), the bounds of the parity tests for these two types (with the
parity tests' allowance of 20 times the operator's own response to inputs changed in their last
bits)."""
import numpy as np
import pytest

from solver_gb300 import configs, frequency, mesher
from solver_gb300.operator import GpuOperator

pytestmark = pytest.mark.gpu

SHAPES = [(1, 2, 1), (2, 1, 3), (3, 2, 2), (2, 4, 1), (5, 3, 2), (3, 8, 2), (9, 7, 3), (15, 16, 1),
          (17, 31, 2), (33, 32, 5), (62, 64, 1), (65, 63, 2), (127, 3, 2), (3, 128, 2),
          (129, 4, 1), (2, 130, 3), (255, 2, 2), (2, 254, 1)]


@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_line_passes(shape):
    cu = np.ones(shape, dtype=bool)
    ax = int(np.argmax(shape))
    b = [0, 0, 0]
    b[ax] = shape[ax] - 1
    req = configs.make_request({"copper": cu}, [dict(configs.COPPER)], (5e-5, 4e-5, 3e-5),
                               [((0, 0, 0), tuple(b))], [1e9], 1e-8)
    out, freqs, _settings, z0, _grid = mesher.parse_request(req)
    esc, inc, cc, diag, exp, ports, le, _li, Zs = out
    op = GpuOperator(inc, exp, diag["P"])
    try:
        op.fill(cc["origin"], cc["sx"], cc["sy"], cc["sz"], esc["Lp"], esc["P"])
        fs = frequency.FrequencyState(2 * np.pi * freqs[0] * esc["freq"], esc, inc, diag, Zs, le,
                                      ports, z0)
        op.set_frequency(fs.w, fs.DZ, fs.Yle, fs.lu)
        rng = np.random.default_rng(4)
        x = rng.standard_normal(op.N) + 1j * rng.standard_normal(op.N)
        ref = op.matvec(x, 0)
        peak = np.max(np.abs(ref))
        noise = np.max(np.abs(op.matvec(x * (1 + np.finfo(float).eps * rng.choice([-1, 1], op.N)), 0)
                              - ref)) / peak
        y = op.matvec(x, 1)
        assert np.max(np.abs(y - ref)) < 2e-5 * peak
        assert np.array_equal(op.matvec(x, 1), y)
        assert np.max(np.abs(op.matvec(x, 2) - ref)) < max(1e-11, 20 * noise) * peak
    finally:
        op.close()
