"""GPU: the near-field fill from corner tables (fill.cu) at the sizes where the tables change
form -- single cells and unit axes, cells whose edges round differently along each axis (few
shared corners), an origin off zero, and a grid whose tables take several slabs of cells --
against the oracle's direct sums: every entry within 64 eps of its sum of |terms|, the bound
of the far-field fill tests."""
import numpy as np
import pytest

from oracle import peec_oracle as O
from solver_gb300 import configs, mesher

pytestmark = pytest.mark.gpu

GRIDS = [((2, 1, 1), (1e-4, 1e-4, 1e-4), 0.0), ((1, 3, 2), (1e-4, 2e-4, 1e-5), 0.0),
         ((5, 1, 7), (3.7e-5, 6.2e-5, 1.85e-5), 1.1e-3), ((17, 9, 5), (1.23e-5, 4.7e-5, 3.1e-5), -2e-3),
         ((33, 20, 3), (5e-4, 2.5e-3, 2.4e-5), 0.0), ((112, 112, 56), (5e-5, 5e-5, 5e-5), 0.0)]


@pytest.mark.parametrize("shape,cell,origin", GRIDS)
def test_fill_matches_oracle(shape, cell, origin):
    from solver_gb300.operator import GpuOperator
    cu = np.zeros(shape, dtype=bool)
    ax = int(np.argmax(shape))
    a, b = [0, 0, 0], [0, 0, 0]
    b[ax] = 1
    cu[tuple(a)] = cu[tuple(b)] = True
    req = configs.make_request({"copper": cu}, [dict(configs.COPPER)], cell,
                               [(tuple(a), tuple(b))], [1e9], 1e-8)
    req["mesherOutput"]["origin"] = {"origin_x": origin, "origin_y": -origin, "origin_z": origin}
    out, _freqs, _settings, _z0, grid = mesher.parse_request(req)
    esc, inc, cc, diag, exp = out[0], out[1], out[2], out[3], out[4]
    ref = O.fill_rows(cc, esc, *grid, with_scale=True)
    op = GpuOperator(inc, exp, diag["P"])
    try:
        got = op.fill(cc["origin"], cc["sx"], cc["sy"], cc["sz"], esc["Lp"], esc["P"],
                      return_rows=True)
        again = op.fill(cc["origin"], cc["sx"], cc["sy"], cc["sz"], esc["Lp"], esc["P"],
                        return_rows=True)
    finally:
        op.close()
    eps = np.finfo(float).eps
    for key, (row, scale) in ref.items():
        if not np.size(row):
            continue
        assert np.all(np.abs(got[key] - row) <= 64 * eps * scale + 1e-300), key
        assert np.array_equal(got[key], again[key]), key


@pytest.mark.parametrize("shape,cell", [((270, 3, 2), (5e-5, 5e-5, 5e-5)),
                                        ((3, 2, 120), (4e-5, 6e-5, 1.2e-4)),
                                        ((2, 190, 40), (2e-4, 3e-5, 4e-5)),
                                        ((40, 30, 3), (1e-3, 1e-3, 1.1e-6)),
                                        ((40, 30, 3), (1e-3, 1e-3, 1.3e-6))])
def test_fill_near_far_boundary(shape, cell):
    """The near-field test by distance (fill.cu, near_for_sure) around its bound, where cells go
    from one test to the other and then to the far field: rows far longer than 166 cells along
    each axis, uneven cells, and cells at the shape (1.2e-3) beyond which it is not used."""
    test_fill_matches_oracle(shape, cell, 0.0)
