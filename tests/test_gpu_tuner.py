"""GPU: the tuner of the FP32 z passes times each kernel form once. "direct_yz" is another name of
"direct": it is no candidate, so it is neither timed nor picked, and pinning it runs the direct
kernels."""
import numpy as np
import pytest

from solver_gb300 import configs, frequency, mesher
from solver_gb300.operator import GpuOperator

pytestmark = pytest.mark.gpu


def test_forms_timed_once():
    req = configs.random_mixed((30, 26, 20), s=5e-5, p=0.4, seed=8, nports=1, freqs=[1e9], tol=1e-8)
    out, freqs, _s, z0, _grid = mesher.parse_request(req)
    esc, inc, cc, diag, exp, ports, le, _li, Zs = out
    op = GpuOperator(inc, exp, diag["P"])
    try:
        op.fill(cc["origin"], cc["sx"], cc["sy"], cc["sz"], esc["Lp"], esc["P"])
        t = op.zpass_tuning()
        assert t["face_ms"]["direct_yz"] is None and t["face_ms"]["staged"] is not None, t
        assert all(t["edge_ms"][f"plan{p}_direct_yz"] is None for p in (0, 1)), t
        assert all(t["edge_ms"][f"plan{p}_direct"] is not None for p in (0, 1)), t
        assert "direct_yz" not in (t["face"], t["edge"])
        fs = frequency.FrequencyState(2 * np.pi * freqs[0] * esc["freq"], esc, inc, diag, Zs, le,
                                      ports, z0)
        op.set_frequency(fs.w, fs.DZ, fs.Yle, fs.lu)
        x = np.random.default_rng(1).standard_normal(op.N) + 0j
        y = []
        for form in ("direct", "direct_yz"):
            op.set_zpass_forms(form, form)
            y.append(op.matvec(x, 1))
        assert np.array_equal(*y)
    finally:
        op.close()
