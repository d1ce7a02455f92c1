"""An upload right after cueva_download_async.  Above 4 MB of primitives each
field goes back up as soon as it has come down (14 copies, one wait per
field); smaller pinned grids go up in one launch (k_upload_begin) after the
whole readback.  Which of the two ran is read from the runtime calls; either
way the state and the arrays are those of the synchronous loop."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PRIMS = ["rho", "p", "vx", "vy", "vz", "psi", "phi", "Ex", "Ey", "Ez", "Bx", "By", "Bz", "q"]


def make(imax, jmax, pinned=True):
    from cueva import Cueva
    g = Cueva(imax, jmax, flux_solver=7, rec_mp=0, sigma=1e3, pinned=pinned)
    g.kh_init(v0=0.5, a=0.05)
    return g


def upload_calls(g):
    """2D copies of one upload, and kernel launches (k_upload_begin, or
    k_begin_step after copies)"""
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        g.upload()
        g.sync()
    counts = {e.key: e.count for e in prof.key_averages()}
    return counts.get("cudaMemcpy2DAsync", 0), counts.get("cudaLaunchKernel", 0)


# 112 bytes a point: 0.7, 3.7, 5.1, 9.0 and 13.5 MB
@pytest.mark.parametrize("imax,jmax,pending,idle", [(96, 64, 0, 0), (256, 128, 0, 0), (300, 150, 14, 0),
                                                    (400, 200, 14, 0), (400, 300, 14, 14)])
def test_fields_go_up_as_they_come_down(imax, jmax, pending, idle):
    g = make(imax, jmax)
    assert upload_calls(g) == (idle, 1)
    g.step(1)
    g.download_async()
    assert upload_calls(g) == (pending, 1)
    g.step(1)
    g.download_async()
    g.sync()
    g.close()


@pytest.mark.parametrize("imax,jmax", [(256, 128), (300, 150), (340, 300), (403, 201)])
@pytest.mark.parametrize("pinned", [True, False])
def test_loop_equals_synchronous(imax, jmax, pinned):
    a, b = make(imax, jmax, pinned), make(imax, jmax, pinned)
    for _ in range(4):
        a.upload()
        a.step(1)
        a.download()
    for _ in range(4):
        b.upload()
        b.step(1)
        b.download_async()
    b.sync()
    for n in PRIMS:
        assert np.array_equal(a.array(n), b.array(n)), n
    a.close()
    b.close()
