"""GPU: the pair z passes (fftconv_impl.cuh, k_zpair and k_zpair_wide) at every circulant
length they take along z (2 to 128 points, where the split of a column over threads changes)
and just above, with every row of the half occupied or few of them, fewer columns than a CTA
takes, ragged x and y extents and absent edge families.

The FP32 pair form and the float-float operator against the FP64 one, whose z passes are the
direct kernels: 2e-5 and 1e-11 relative (max-norm), the bounds of the parity tests for these
two types (with the parity tests' allowance of 20 times the operator's own response to inputs
changed in their last bits), and the FP32 direct form to the same bound, so that a fault of either form shows."""
import numpy as np
import pytest

from solver_gb300 import configs, frequency, mesher
from solver_gb300.operator import GpuOperator

pytestmark = pytest.mark.gpu

SHAPES = [(3, 2, 1), (2, 5, 2), (9, 4, 3), (1, 6, 4), (5, 33, 5), (6, 1, 8), (13, 3, 15),
          (3, 4, 16), (40, 3, 17), (5, 2, 31), (2, 3, 32), (4, 2, 33), (2, 2, 62), (3, 2, 63),
          (2, 7, 64)]


@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_pair_forms(shape):
    cu = np.ones(shape, dtype=bool)
    ax = int(np.argmax(shape))
    a, b = [0, 0, 0], [0, 0, 0]
    b[ax] = shape[ax] - 1
    req = configs.make_request({"copper": cu}, [dict(configs.COPPER)], (5e-5, 4e-5, 3e-5),
                               [(tuple(a), tuple(b))], [1e9], 1e-8)
    out, freqs, _settings, z0, grid = mesher.parse_request(req)
    esc, inc, cc, diag, exp, ports, le, _li, Zs = out
    op = GpuOperator(inc, exp, diag["P"])
    try:
        op.fill(cc["origin"], cc["sx"], cc["sy"], cc["sz"], esc["Lp"], esc["P"])
        fs = frequency.FrequencyState(2 * np.pi * freqs[0] * esc["freq"], esc, inc, diag, Zs, le,
                                      ports, z0)
        op.set_frequency(fs.w, fs.DZ, fs.Yle, fs.lu)
        rng = np.random.default_rng(3)
        x = rng.standard_normal(op.N) + 1j * rng.standard_normal(op.N)
        ref = op.matvec(x, 0)
        peak = np.max(np.abs(ref))
        noise = np.max(np.abs(op.matvec(x * (1 + np.finfo(float).eps * rng.choice([-1, 1], op.N)), 0)
                              - ref)) / peak
        Lz = [f["L"][2] for f in op.conv_info()]
        for form in ("pair", "direct"):
            op.set_zpass_forms(form, form)
            t = op.zpass_tuning()
            assert t["face"] == (form if Lz[0] <= 128 else "direct"), (t, Lz)
            y = op.matvec(x, 1)
            assert np.max(np.abs(y - ref)) < 2e-5 * peak, form
            assert np.array_equal(op.matvec(x, 1), y)
        assert np.max(np.abs(op.matvec(x, 2) - ref)) < max(1e-11, 20 * noise) * peak
    finally:
        op.close()
