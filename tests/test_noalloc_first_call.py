"""The first call of the allocation-free Poisson solve in a process, on a non-blocking stream: everything it
reads is in place whichever stream makes it and whatever the copy engines are doing."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import ctypes, sys
sys.path.insert(0, %r)
sys.path.insert(0, %r)
import numpy as np, torch
import hipace2_b200 as hp
from test_fft_dst_lengths import dense

n = %d
L = hp.load_library()
f = np.random.default_rng(n).standard_normal((n, n))
ft = torch.from_numpy(f).cuda()
u = torch.full_like(ft, float("nan"))
src = torch.empty(1 << 28, dtype=torch.uint8).pin_memory()
dst = torch.empty(1 << 28, dtype=torch.uint8, device="cuda")
busy, s = torch.cuda.Stream(), torch.cuda.Stream()
torch.cuda.synchronize()
with torch.cuda.stream(busy):
    for _ in range(4):
        dst.copy_(src, non_blocking=True)  # uploads in flight during the call
rc = L.hpq_poisson_dirichlet_noalloc(ft.data_ptr(), u.data_ptr(), n, n, 0.11, 0.07, ctypes.c_void_p(s.cuda_stream))
torch.cuda.synchronize()
want = dense(f, 0.11, 0.07)
err = np.linalg.norm(u.cpu().numpy() - want) / np.linalg.norm(want)
print(rc, err)
# four transforms of log2(2(n+1)) <= 11 levels, a few roundings of 1.1e-16 each
assert rc == 0 and err <= 4 * 11 * 4 * 1.1e-16, (rc, err)
"""


@pytest.mark.parametrize("n", [31, 255, 1023])
def test_first_call_on_a_non_blocking_stream(n):
    r = subprocess.run([sys.executable, "-c", SCRIPT % (ROOT, os.path.join(ROOT, "tests"), n)], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("nx,ny", [(31, 63), (1023, 255)])
def test_captured_solve_replays_on_new_right_hand_sides(nx, ny):
    import ctypes

    import numpy as np
    import torch

    import hipace2_b200 as hp
    from test_fft_dst_lengths import dense

    L = hp.load_library()
    rng = np.random.default_rng(nx)
    ft = torch.zeros((ny, nx), dtype=torch.float64, device="cuda")
    u, w = torch.full_like(ft, float("nan")), torch.full_like(ft, float("nan"))

    def solve(f, out):
        s = torch.cuda.current_stream().cuda_stream
        assert L.hpq_poisson_dirichlet_noalloc(f.data_ptr(), out.data_ptr(), nx, ny, 0.11, 0.07, ctypes.c_void_p(s)) == 0

    solve(ft, u)  # (the first call on a device precedes any capture)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        solve(ft, u)
        ft.mul_(2.0)  # a kernel of the caller behind the solve, then another solve
        solve(ft, w)
    for _ in range(3):
        f = rng.standard_normal((ny, nx))
        ft.copy_(torch.from_numpy(f))
        graph.replay()
        torch.cuda.synchronize()
        want = dense(f, 0.11, 0.07)
        bound = 4 * 11 * 4 * 1.1e-16 * np.linalg.norm(want)
        assert np.linalg.norm(u.cpu().numpy() - want) <= bound
        assert np.linalg.norm(w.cpu().numpy() - 2 * want) <= 2 * bound
