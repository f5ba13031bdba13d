"""What the multigrid tolerance means in single precision: the fields that a converged solve returns satisfy the
equation to the tolerance, up to the rounding of a solution stored in 32 bits. Evaluated here in 64 bits from the
slice's own right-hand side, coefficient and fields."""
import numpy as np
import pytest

import hipace2_b200 as hp
from cases import EXPLICIT_MOVING

pytestmark = pytest.mark.gpu


def residual(u, rhs, chi, dx, dy, cell):
    """rhs + chi u - Lap u, zero one cell outside (node-centred) or on the faces (cell-centred)"""
    p = np.pad(u, 1)
    h, v = p[1:-1, :-2] + p[1:-1, 2:], p[:-2, 1:-1] + p[2:, 1:-1]
    cx, cy = np.full(u.shape, 2.0), np.full(u.shape, 2.0)
    if cell:
        h[:, [0, -1]] *= 4 / 3
        v[[0, -1], :] *= 4 / 3
        cx[:, [0, -1]] = 4
        cy[[0, -1], :] = 4
    diag = cx / dx ** 2 + cy / dy ** 2 + chi
    return rhs + diag * u - h / dx ** 2 - v / dy ** 2, diag


# clusters and tiles, node- and cell-centred, flat cells; 1e-4 in single precision throughout, 1e-8 refined
@pytest.mark.parametrize("nx,ny", [(255, 255), (511, 63), (63, 511), (256, 256), (511, 511), (512, 512), (767, 383)])
@pytest.mark.parametrize("tol", [1e-4, 1e-8])
def test_residual_of_the_returned_fields(nx, ny, tol):
    text = (EXPLICIT_MOVING.replace("amr.n_cell = 33 33 40", "amr.n_cell = %d %d 12" % (nx, ny))
            .replace("hipace.MG_tolerance_rel = 1e-12", "hipace.MG_tolerance_rel = %g" % tol)
            .replace("beam.density = 5.", "beam.density = 0.05"))
    sim = hp.Hipace(text, precision=hp.MIXED, graphs=False)
    sim.init_data()
    sim.begin_step(0)
    for s in range(11, -1, -1):
        sim.solve_one_slice(s)
        if s not in (7, 4):
            continue
        chi, dx, dy = sim.get_field("chi"), 12.0 / nx, 12.0 / ny
        for b, r in (("Bx", "Sy"), ("By", "Sx")):
            u, rhs = sim.get_field(b), sim.get_field(r)
            res, diag = residual(u, rhs, chi, dx, dy, nx % 2 == 0)
            scale = max(np.abs(sim.get_field(k)).max() for k in ("Sx", "Sy"))
            assert scale > 0
            # rounding of the stored solution and of the last sweep: half a unit each in the point and in the sum of its
            # neighbours, 6e-8 of |u|, times the diagonal
            stored = 4 * 6e-8 * (diag * np.abs(u)).max()
            assert np.abs(res).max() <= 1.01 * tol * scale + stored, (s, b, np.abs(res).max() / scale, stored / scale)
    sim.end_step()
    sim.close()
