"""Creating a context or an ensemble sets up (and thereby loads) the kernels
that its grids run: the wide form of the stage kernel only on small grids.
Counted from the runtime calls: the y-face kernel and the three x-face
kernels for two tile heights, two ring kernels where the ring exists (MP5 and
the MC slopes), two wide kernels on small grids of flux routines 5-7."""
import pytest

pytestmark = pytest.mark.gpu


def attribute_calls(make):
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        obj = make()
    obj.close()
    return {e.key: e.count for e in prof.key_averages()}.get("cudaFuncSetAttribute", 0)


@pytest.mark.parametrize("imax,jmax,solver,rec,expected", [
    (64, 32, 5, 0, 12), (64, 32, 7, 2, 10), (64, 32, 2, 0, 10),
    (400, 300, 5, 0, 10), (400, 300, 7, 1, 8), (400, 300, 2, 0, 10),
])
def test_context(imax, jmax, solver, rec, expected):
    from cueva import Cueva
    assert attribute_calls(lambda: Cueva(imax, jmax, flux_solver=solver, rec_mp=rec)) == expected


@pytest.mark.parametrize("sizes,expected", [([(64, 32)] * 3, 12), ([(300, 200)] * 3, 10)])
def test_ensemble(sizes, expected):
    from cueva.ensemble import Ensemble
    kws = [dict(imax=a, jmax=b, order=2, flux_solver=5, rec_mp=0) for a, b in sizes]
    assert attribute_calls(lambda: Ensemble(kws)) == expected


def test_ensemble_returns_to_the_wide_form():
    """tiles of 4 rows (no wide form) and back: the kernels are set up"""
    import numpy as np
    from cueva.ensemble import Ensemble
    out = []
    for shapes in ((), ((4, 0), (8, 0))):
        ens = Ensemble([dict(imax=60, jmax=33, order=2, flux_solver=7, rec_mp=1, sigma=1e3)])
        for rows, ctas in shapes:
            ens.set_shape(rows=rows, ctas_per_sm=ctas)
        ens.kh_init(0, v0=0.5, a=0.05)
        ens.step(2)
        ens.sync()
        out.append(ens.get_prims(0))
        ens.close()
    for n in out[0]:
        assert np.array_equal(out[0][n], out[1][n]), n
