"""GPU: operator applications whose output is, or overlaps, their input (peec_matvec_dev). The final
rows read x after the groups have written y's node block, so such an application works on a copy of
x; it gives the bits of one between separate vectors, in every arithmetic, on its first call and on
later ones (captured graphs), and after the frequency state was replaced."""
import numpy as np
import pytest
import torch

from solver_gb300 import configs, frequency, mesher
from solver_gb300.operator import GpuOperator

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def system():
    req = configs.random_mixed((13, 11, 7), s=5e-5, p=0.5, seed=3, nports=1, freqs=[1e9], tol=1e-8)
    out, freqs, _s, z0, _grid = mesher.parse_request(req)
    esc, inc, cc, diag, exp, ports, le, _li, Zs = out
    op = GpuOperator(inc, exp, diag["P"])
    op.fill(cc["origin"], cc["sx"], cc["sy"], cc["sz"], esc["Lp"], esc["P"])
    states = [frequency.FrequencyState(2 * np.pi * f * esc["freq"], esc, inc, diag, Zs, le, ports, z0)
              for f in (freqs[0], 2.5 * freqs[0])]
    yield op, states
    op.close()


@pytest.mark.parametrize("prec", [0, 1, 2])
def test_output_over_its_input(system, prec):
    op, states = system
    N = op.N
    rng = np.random.default_rng(prec)
    x = torch.from_numpy(rng.standard_normal(N) + 1j * rng.standard_normal(N)).cuda()
    buf = torch.empty(3 * N, dtype=torch.complex128, device="cuda")
    size = 16
    for fs in states:
        op.set_frequency(fs.w, fs.DZ, fs.Yle, fs.lu)
        ref = torch.empty_like(x)
        torch.cuda.synchronize()
        op.matvec_dev(x.data_ptr(), ref.data_ptr(), prec)
        for shift in (0, 1, -1, N // 3, -(op.m + 1), N - 1, N):
            for _ in range(3):
                buf.fill_(7.0)
                buf[N:2 * N] = x
                torch.cuda.synchronize()
                at = buf.data_ptr() + size * N
                op.matvec_dev(at, at + size * shift, prec)
                assert torch.equal(buf[N + shift:2 * N + shift], ref), shift
