"""Accuracy of the single-precision multigrid: on fine grids the weights of a sweep, rounded to 32 bits, would
shift the coefficient chi by up to 6e-8 * 4 / dx^2 (4e-4 here), and the fields with it."""
import numpy as np
import pytest

import hipace2_b200 as hp
from cases import EXPLICIT_MOVING

pytestmark = pytest.mark.gpu


def run(nx, ny, tol):
    text = (EXPLICIT_MOVING.replace("amr.n_cell = 33 33 40", "amr.n_cell = %d %d 12" % (nx, ny))
            .replace("hipace.MG_tolerance_rel = 1e-12", "hipace.MG_tolerance_rel = %g" % tol)
            .replace("beam.density = 5.", "beam.density = 0.05"))
    g = hp.Hipace(text, precision=hp.MIXED, deterministic=True)
    g.init_data()
    g.set_diag(["Bx", "By"])
    g.step(0)
    out = {k: g.get_diag(k) for k in ("Bx", "By")}
    g.close()
    return out


# cluster form and tiles; node-centred grids, where a V-cycle reduces an error 30 times, so that the tolerance
# does not hide the rounding (cell-centred ones, 0.4 per V-cycle, end with 1e-4 of the slowest modes left)
@pytest.mark.parametrize("nx,ny", [(511, 63), (63, 511), (511, 511), (767, 383)])
def test_single_precision_solve_against_refined(nx, ny):
    a = run(nx, ny, 1e-4)
    b = run(nx, ny, 1e-8)  # the same arrays, solved with a solution and residual in 64 bits
    for k in a:
        # chi of about 1 bounds the smallest eigenvalue: an error is at most about the residual, 1e-4
        assert np.linalg.norm(a[k] - b[k]) <= 1e-4 * np.linalg.norm(b[k]), k
