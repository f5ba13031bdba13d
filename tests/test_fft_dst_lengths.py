"""The register FFT of the DST-I (radix-8 passes, then one of radix 8, 4 or 2) at every length it is
compiled for, against dense sine matrices: M = 64 .. 2048 through the allocation-free Poisson solve
(double), M = 64 .. 4096 and the Bluestein lengths L = 64 .. 8192 in both precisions through the
slice loop's Psi solve."""
import ctypes

import numpy as np
import pytest

import hipace2_b200 as hp

pytestmark = pytest.mark.gpu


def dense(f, dx, dy):
    ny, nx = f.shape

    def sine(n):
        k = np.arange(1, n + 1)
        return np.sin(np.outer(k, k) * np.pi / (n + 1)), np.sin(k * np.pi / (2 * (n + 1))) ** 2

    sx, ex = sine(nx)
    sy, ey = sine(ny)
    eig = -4 * (ey[:, None] / dy ** 2 + ex[None, :] / dx ** 2)
    return sy @ ((sy @ f @ sx) * (4.0 / ((nx + 1) * (ny + 1))) / eig) @ sx


@pytest.mark.parametrize("nx,ny", [(31, 31), (63, 127), (127, 31), (255, 63), (511, 255), (1023, 511), (31, 1023), (1023, 1023)])
def test_poisson_at_every_length(nx, ny):
    import torch
    rng = np.random.default_rng(nx * 2000 + ny)
    f = rng.standard_normal((ny, nx))
    dx, dy = 0.11, 0.07
    ft = torch.from_numpy(f).cuda()
    u = torch.full_like(ft, np.nan)  # every element is written
    L = hp.load_library()
    for stream in (None, torch.cuda.Stream()):
        with torch.cuda.stream(stream) if stream else torch.cuda.stream(torch.cuda.current_stream()):
            u.fill_(np.nan)
            torch.cuda.synchronize()
            s = torch.cuda.current_stream().cuda_stream
            assert L.hpq_poisson_dirichlet_noalloc(ft.data_ptr(), u.data_ptr(), nx, ny, dx, dy, ctypes.c_void_p(s)) == 0
            torch.cuda.synchronize()
        want = dense(f, dx, dy)
        # four transforms of log2(2(n+1)) <= 11 levels, a few roundings of 1.1e-16 each
        assert np.linalg.norm(u.cpu().numpy() - want) <= 4 * 11 * 4 * 1.1e-16 * np.linalg.norm(want)


def smallest_eigenvalue(nx, ny, dx, dy):
    return 4 * (np.sin(np.pi / (2 * (nx + 1))) ** 2 / dx ** 2 + np.sin(np.pi / (2 * (ny + 1))) ** 2 / dy ** 2)


# radix-2 axes: M = 2(n + 1); Bluestein axes: L >= 4(n + 1) - 1, 64 128 256 512 1024 2048 4096 8192; each length on
# the x axis (first and last pass) and on the y axis (eigenvalue pass)
@pytest.mark.parametrize("nx,ny", [(31, 63), (127, 31), (63, 255), (255, 127), (511, 1023), (1023, 511), (2047, 31), (31, 2047),
                                   (14, 20), (20, 14), (40, 100), (100, 40), (250, 320), (320, 250), (600, 1200), (1200, 600),
                                   (2046, 34), (321, 63), (255, 41)])
@pytest.mark.parametrize("precision", [hp.PLAIN_FP64, hp.MIXED])
def test_psi_at_every_length_and_precision(nx, ny, precision, monkeypatch):
    from cases import PC_SMALL
    monkeypatch.setenv("HPQ_DST", "fft")  # (in single precision the default on some of these grids are the sine GEMMs)
    text = (PC_SMALL.replace("amr.n_cell = 32 32 40", "amr.n_cell = %d %d 8" % (nx, ny))
            .replace("beam.position_mean = 0. 0. 0.", "beam.position_mean = 0.7 -0.4 0."))
    sim = hp.Hipace(text, precision=precision, graphs=False)
    sim.init_data()
    sim.begin_step(0)
    for s in range(7, 3, -1):
        sim.solve_one_slice(s)
    f, psi = -sim.get_field("rhomjz"), sim.get_field("Psi")
    for s in range(3, -1, -1):
        sim.solve_one_slice(s)
    sim.end_step()
    sim.close()
    dx, dy = 16.0 / nx, 16.0 / ny
    want = dense(f, dx, dy)
    assert np.linalg.norm(want) > 0
    # four transforms, each of at most two FFTs of 13 levels and three products, two roundings a step; what they add
    # to the lowest mode is divided by the smallest eigenvalue
    eps = 1.1e-16 if precision == hp.PLAIN_FP64 else 6e-8
    bound = 4 * 29 * 2 * eps * max(np.linalg.norm(want), np.linalg.norm(f) / smallest_eigenvalue(nx, ny, dx, dy))
    assert np.linalg.norm(psi - want) <= bound, (np.linalg.norm(psi - want) / np.linalg.norm(want), bound / np.linalg.norm(want))
