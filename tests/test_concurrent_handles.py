"""Several handles on one GPU, each driven by its own host thread: the multigrid clusters of all handles together
need more room than the GPU has, and each solve's two clusters wait for each other's norms."""
import threading

import numpy as np
import pytest

import hipace2_b200 as hp

pytestmark = pytest.mark.gpu


def handle(nx, precision):
    from cases import EXPLICIT_MOVING
    text = (EXPLICIT_MOVING.replace("amr.n_cell = 33 33 40", "amr.n_cell = %d %d 24" % (nx, nx))
            .replace("hipace.MG_tolerance_rel = 1e-12", "hipace.MG_tolerance_rel = 1e-6"))
    g = hp.Hipace(text, precision=precision, deterministic=True)
    g.init_data()
    g.set_diag(["Bx", "By", "Ez"])
    g.step(0)  # (captures the slice graph, during which CUDA refuses other threads' synchronising calls)
    return g


def fields(g):
    for s in range(1, 5):
        g.step(s)
    out = {k: g.get_diag(k) for k in ("Bx", "By", "Ez")}
    g.close()
    return out


# one block per cluster, clusters of 16
@pytest.mark.parametrize("nx,precision", [(63, hp.PLAIN_FP64), (255, hp.PLAIN_FP64), (255, hp.MIXED)])
def test_handles_on_threads_give_the_results_of_one_alone(nx, precision):
    want = fields(handle(nx, precision))
    handles = [handle(nx, precision) for _ in range(10)]
    got, errors = {}, []

    def work(i):
        try:
            got[i] = fields(handles[i])
        except Exception as e:  # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(10)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for i in range(10):
        for k in want:
            assert np.array_equal(got[i][k], want[k]), (i, k)
