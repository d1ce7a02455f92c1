"""The fused stage kernel's wide form (small grids: one-band tiles of 4 to 12
warps, two fields per limiter call) and its rule (stage_wide_rows): grids on
both sides of every switch, against the two-kernel form, bit for bit -- MP5
through set_stage_kernel, MP7 and MP9 through an ensemble with tiles of 4 rows,
which always runs k_yface + k_xupd."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# imax, jmax: 4 warps on few and on many SMs; the first grids that need 5, 8 and 12;
# the first above (ring form); ragged last strips and segments throughout
GRIDS = [(6, 6), (61, 32), (124, 87), (155, 95), (186, 143), (278, 145), (310, 147), (342, 151), (403, 200)]


def state(imax, jmax):
    rng = np.random.default_rng(imax)
    y, x = np.meshgrid(np.linspace(0, 1, jmax + 1), np.linspace(-1, 1, imax + 1), indexing="ij")
    from cueva import PRIM_FIELDS
    out = {}
    for n in PRIM_FIELDS:
        w = sum(rng.uniform(0.3, 1) * np.sin(2 * np.pi * m * y + rng.uniform(0, 6)) * np.cos(np.pi * m * x + 1)
                for m in (1, 2, 5))
        out[n] = (1.0 if n in ("rho", "p") else 0.0) + 0.03 * w
    out["vy"] = out["vy"] + 0.4 * np.tanh(x / 0.05)
    return out


def run_single(kw, prims, fused=None):
    from cueva import Cueva
    g = Cueva(**kw)
    if fused is not None:
        g.set_stage_kernel(fused)
    for n, a in prims.items():
        g.set_interior(n, a)
    g.upload()
    g.step(2)
    g.download()
    out = {n: g.interior(n).copy() for n in prims}
    g.close()
    return out


@pytest.mark.parametrize("imax,jmax", GRIDS)
@pytest.mark.parametrize("solver,precision", [(5, 0), (6, 0), (7, 0), (7, 1)])
def test_wide_equals_two_kernels_mp5(imax, jmax, solver, precision):
    kw = dict(imax=imax, jmax=jmax, order=2, flux_solver=solver, rec_mp=0, precision=precision, sigma=1e3,
              bc_x=imax % 2)
    prims = state(imax, jmax)
    a, b = run_single(kw, prims, 1), run_single(kw, prims, 0)
    for n in prims:
        assert np.array_equal(a[n], b[n]), n


@pytest.mark.parametrize("imax,jmax", GRIDS)
@pytest.mark.parametrize("rec,precision", [(1, 0), (2, 0), (1, 1), (2, 1)])
def test_wide_equals_two_kernels_mp7_mp9(imax, jmax, rec, precision):
    from cueva.ensemble import Ensemble
    kw = dict(imax=imax, jmax=jmax, order=2, flux_solver=7, rec_mp=rec, precision=precision, sigma=1e3, bc_x=0)
    prims = state(imax, jmax)
    a = run_single(kw, prims)
    ens = Ensemble([kw])
    ens.set_shape(rows=4)
    ens.set_prims(0, prims)
    ens.step(2)
    ens.sync()
    b = ens.get_prims(0)
    ens.close()
    for n in prims:
        assert np.array_equal(a[n], b[n]), n


def test_small_ensemble_runs_the_wide_form_and_equals_single_runs():
    from cueva.ensemble import Ensemble
    kws = [dict(imax=40 + 9 * k, jmax=20 + 3 * k, order=4, intsum_reset=1, flux_solver=7, rec_mp=0, sigma=1e3)
           for k in range(5)]
    ens = Ensemble(kws)
    for k, kw in enumerate(kws):
        ens.set_prims(k, state(kw["imax"], kw["jmax"]))
    ens.step(2)
    ens.sync()
    for k, kw in enumerate(kws):
        a, b = run_single(kw, state(kw["imax"], kw["jmax"])), ens.get_prims(k)
        for n in b:
            assert np.array_equal(a[n], b[n]), (k, n)
    ens.close()
