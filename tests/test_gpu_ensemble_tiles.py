"""Segment heights of the fused stage kernel's tiles (stage_seg_rows).  Grids
on both sides of the heights of one to four bands against the two-kernel form,
and ensembles, whose grids share one height -- unlike and like grids, ragged
strips and segments, few tiles and many waves of them -- against single runs
with each grid's own height, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MIXES = {
    "unlike": [(420, 211), (61, 9), (130, 402), (33, 64), (6, 6), (250, 250)],
    "one large": [(900, 700), (64, 32), (40, 77)],
    "like": [(310, 187)] * 5,
    "many waves": [(620, 611)] * 6 + [(95, 15), (311, 8)],
}


def state(imax, jmax, k):
    from cueva import PRIM_FIELDS
    rng = np.random.default_rng(1000 * imax + jmax + k)
    y, x = np.meshgrid(np.linspace(0, 1, jmax + 1), np.linspace(-1, 1, imax + 1), indexing="ij")
    out = {}
    for n in PRIM_FIELDS:
        w = sum(rng.uniform(0.3, 1) * np.sin(2 * np.pi * m * y + rng.uniform(0, 6)) * np.cos(np.pi * m * x + 1)
                for m in (1, 2, 5))
        out[n] = (1.0 if n in ("rho", "p") else 0.0) + 0.03 * w
    out["vy"] = out["vy"] + 0.4 * np.tanh(x / 0.05)
    return out


@pytest.mark.parametrize("mix", list(MIXES))
@pytest.mark.parametrize("solver,precision", [(7, 0), (5, 1), (1, 0)])
def test_shared_segments_equal_single_runs(mix, solver, precision):
    from cueva import Cueva
    from cueva.ensemble import Ensemble
    kws = [dict(imax=a, jmax=b, order=2, flux_solver=solver, rec_mp=0, precision=precision, sigma=1e3)
           for a, b in MIXES[mix]]
    ens = Ensemble(kws)
    for k, kw in enumerate(kws):
        ens.set_prims(k, state(kw["imax"], kw["jmax"], k))
    ens.step(2)
    ens.sync()
    for k, kw in enumerate(kws):
        g = Cueva(**kw)
        for n, a in state(kw["imax"], kw["jmax"], k).items():
            g.set_interior(n, a)
        g.upload()
        g.step(2)
        g.download()
        b = ens.get_prims(k)
        for n in b:
            assert np.array_equal(g.interior(n), b[n]), (k, n)
        g.close()
    ens.close()


@pytest.mark.parametrize("imax,jmax", [(403, 301), (640, 340), (999, 451), (1003, 777), (1500, 1200), (2200, 1900)])
@pytest.mark.parametrize("solver,precision", [(7, 0), (7, 1)])
def test_segments_equal_two_kernels(imax, jmax, solver, precision):
    from cueva import Cueva
    prims, out = state(imax, jmax, 0), []
    for fused in (1, 0):
        g = Cueva(imax=imax, jmax=jmax, order=2, flux_solver=solver, rec_mp=0, precision=precision, sigma=1e3)
        g.set_stage_kernel(fused)
        for n, a in prims.items():
            g.set_interior(n, a)
        g.upload()
        g.step(2)
        g.download()
        out.append({n: g.interior(n).copy() for n in prims})
        g.close()
    for n in prims:
        assert np.array_equal(out[0][n], out[1][n]), n
