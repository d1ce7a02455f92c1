"""cueva_set_stage_kernel(0) gives the two-kernel form (a y-face launch per
stage, counted by cueva_profile_steps) for every reconstruction, on grids of
the wide form, of the ring and above both; same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PRIMS = ["rho", "p", "vx", "vy", "vz", "psi", "phi", "Ex", "Ey", "Ez", "Bx", "By", "Bz", "q"]


def run(imax, jmax, rec, precision, fused):
    """launches of the y-face kernel in two steps, and the state after them"""
    from cueva import Cueva
    g = Cueva(imax, jmax, order=2, flux_solver=7, rec_mp=rec, precision=precision, sigma=1e3)
    if fused is not None:
        g.set_stage_kernel(fused)
    g.kh_init(v0=0.5, a=0.05)
    g.upload()
    _, launches = g.profile_steps(2)
    g.download()
    out = {n: g.interior(n).copy() for n in PRIMS}
    g.close()
    return launches[0], out


@pytest.mark.parametrize("imax,jmax,small", [(64, 32, True), (220, 196, True), (300, 240, False)])
@pytest.mark.parametrize("rec", [0, 1, 2])
@pytest.mark.parametrize("precision", [0, 1])
def test_zero_runs_two_kernels(imax, jmax, small, rec, precision):
    n0, a = run(imax, jmax, rec, precision, 0)
    n1, b = run(imax, jmax, rec, precision, None)
    assert n0 == 4   # two steps of two stages
    assert n1 == (0 if small or rec == 0 else 4)
    for n in PRIMS:
        assert np.array_equal(a[n], b[n]), n


def test_answers_and_refusals_stay():
    from cueva import Cueva, CuevaError
    g = Cueva(64, 32, order=2, flux_solver=7, rec_mp=2)
    assert g.stage_kernel() == 0
    g.set_stage_kernel(0)
    assert g.stage_kernel() == 0
    with pytest.raises(CuevaError):
        g.set_stage_kernel(1)
    g.close()
    g = Cueva(64, 32, order=2, flux_solver=7, rec_mp=0)
    for fused in (0, 1):
        g.set_stage_kernel(fused)
        assert g.stage_kernel() == fused
    g.close()
