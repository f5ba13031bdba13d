"""The cluster-resident multigrid (grids that fit the shared memory of one thread-block cluster per
component) against the tile form of the same solve (HPQ_MG=tiles): the same colour sweeps, so the same
V-cycles and, up to the rounding of sums taken in another order, the same fields."""
import os

import numpy as np
import pytest

import hipace2_b200 as hp

pytestmark = pytest.mark.gpu


def deck(nx, ny, tol):
    from cases import EXPLICIT_MOVING
    return (EXPLICIT_MOVING.replace("amr.n_cell = 33 33 40", "amr.n_cell = %d %d 12" % (nx, ny))
            .replace("hipace.MG_tolerance_rel = 1e-12", "hipace.MG_tolerance_rel = %g" % tol)
            # a weak (linear) wake: the march does not amplify rounding from slice to slice
            .replace("beam.density = 5.", "beam.density = 0.05"))


def run(text, precision, form):
    old = os.environ.get("HPQ_MG")
    os.environ["HPQ_MG"] = form
    try:
        g = hp.Hipace(text, precision=precision, deterministic=True)
        g.init_data()
    finally:
        os.environ.pop("HPQ_MG", None)
        if old is not None:
            os.environ["HPQ_MG"] = old
    g.set_diag(["Bx", "By", "Ez"])
    g.step(0)
    out = {k: g.get_diag(k) for k in ("Bx", "By", "Ez")}
    cycles = g.counters()["mg_vcycles"]
    g.close()
    return out, cycles


# one block per component (63^2 and below in double) and clusters of 16; rows per thread 1, 2, 4, 8;
# node- and cell-centred; blocks without rows, odd row counts, coarsest levels of a few and of many
# points (matrix of the smallest levels or not), non-square grids
@pytest.mark.parametrize("nx,ny", [(31, 31), (33, 33), (63, 63), (64, 64), (127, 127), (95, 79), (255, 255),
                                   (256, 256), (255, 31), (31, 255), (100, 72), (223, 159), (511, 63), (160, 96)])
@pytest.mark.parametrize("precision,tol", [(hp.PLAIN_FP64, 1e-4), (hp.PLAIN_FP64, 1e-11), (hp.MIXED, 1e-4),
                                           (hp.MIXED, 1e-8)])
def test_cluster_form_equals_tile_form(nx, ny, precision, tol):
    text = deck(nx, ny, tol)
    a, ca = run(text, precision, "cluster")
    b, cb = run(text, precision, "tiles")
    # a V-cycle more or less where a norm meets the target to rounding
    assert cb > 0 and abs(ca - cb) <= max(1, cb // 20), (ca, cb)
    # rounding of a residual, eps 4/dx^2 |B|, against the smallest eigenvalue of the 12 x 12 box, 2 pi^2/144,
    # in each of 12 slices; a V-cycle more or less changes a solution by the tolerance
    dx = 12.0 / max(nx, ny)
    bound = 12 * (1.1e-16 if precision == hp.PLAIN_FP64 else 6e-8) * 4 / dx ** 2 / (2 * np.pi ** 2 / 144)
    if ca != cb:
        bound += 12 * tol
    for k in a:
        assert np.isfinite(a[k]).all()
        assert np.linalg.norm(a[k] - b[k]) <= bound * np.linalg.norm(b[k]), k


# every level split over the cluster: cell-centred, and node-centred with an even number of rows on the coarsest
# level (a finer level has one row more than twice as many)
@pytest.mark.parametrize("nx,ny,tol", [(194, 194, 1e-4), (226, 150, 1e-4), (263, 263, 1e-4), (193, 193, 0.05), (257, 257, 0.05),
                                       (257, 193, 0.05), (321, 65, 0.05), (65, 321, 0.05)])
@pytest.mark.parametrize("precision", [hp.PLAIN_FP64, hp.MIXED])
def test_grids_whose_levels_are_all_split(nx, ny, tol, precision):
    test_cluster_form_equals_tile_form(nx, ny, precision, tol)


# flat grids: blocks own more rows than the grid has, over a coarse level that lies in block 0
@pytest.mark.parametrize("nx,ny", [(587, 31), (571, 31)])
@pytest.mark.parametrize("precision", [hp.PLAIN_FP64, hp.MIXED])
def test_flat_grids_with_rows_beyond_the_grid(nx, ny, precision):
    test_cluster_form_equals_tile_form(nx, ny, precision, 0.3)


def test_profile_counts_the_coefficients_in_the_multigrid_class(monkeypatch):
    text = deck(63, 63, 1e-4)
    for form, slices in (("cluster", 12), ("tiles", 0)):
        monkeypatch.setenv("HPQ_MG", form)
        g = hp.Hipace(text, graphs=False)
        g.init_data()
        g.step(0)
        g.set_profiling(True)
        g.step(1)
        mg, n = g.profile("multigrid")
        coef, m = g.profile("multigrid_coefficients")
        assert n == 12 and m == slices and mg > coef >= 0 and (coef > 0) == (slices > 0)
        g.close()
