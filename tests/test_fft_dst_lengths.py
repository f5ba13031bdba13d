"""The register FFT of the DST-I (radix-8 passes, then one of radix 8, 4 or 2) at every length it is
compiled for, through the allocation-free Poisson solve against dense sine matrices."""
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
