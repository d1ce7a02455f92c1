"""The limiting steps of the MP reconstruction (mp_lim_pair, mp_quad,
cueva_mp.cuh), which smooth data hardly reaches: white noise, steps and single
spikes of every field send most faces there, in every combination of failed
sides.  The stage right-hand side equals the oracle's bit for bit, through
MP5 / MP7 / MP9 and the three flux routines that use them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rough(kind, shape, rng):
    if kind == "noise":
        return rng.uniform(-1.0, 1.0, shape)
    if kind == "steps":
        return np.where((np.add.outer(np.arange(shape[0]) // 3, np.arange(shape[1]) // 4)) % 2 == 0, 1.0, -1.0)
    a = np.zeros(shape)
    a[rng.integers(0, shape[0], 60), rng.integers(0, shape[1], 60)] = rng.uniform(-1.0, 1.0, 60)
    return a


@pytest.mark.parametrize("kind", ["noise", "steps", "spikes"])
@pytest.mark.parametrize("rec", [0, 1, 2])
@pytest.mark.parametrize("solver", [5, 6, 7])
def test_rough_fields_bit_identical(oracle_mod, solver, rec, kind):
    from cueva import PRIM_FIELDS, RHS_FIELDS, STAGE_FIELDS, Cueva
    imax, jmax = 65, 34
    rng = np.random.default_rng(10 * rec + solver)
    shape = (jmax + 1, imax + 1)
    kw = dict(order=2, flux_solver=solver, rec_mp=rec, c2p=1, bc_x=0, bc_y=1, sigma=1e2)
    scale = dict(rho=(1.0, 0.6), p=(1.0, 0.6), vx=(0.0, 0.2), vy=(0.0, 0.2), vz=(0.0, 0.2))
    prims = {n: scale.get(n, (0.0, 0.1))[0] + scale.get(n, (0.0, 0.1))[1] * rough(kind, shape, rng)
             for n in PRIM_FIELDS}
    oracle_mod.set_libm_seed(0)
    o = oracle_mod.Oracle(imax, jmax, **kw)
    o.set_prims(prims)
    o.run_stages(1)
    g = Cueva(imax, jmax, **kw)
    for n in STAGE_FIELDS[:17]:
        g.set_interior(n, o.named(n), 1)
    for n in prims:
        g.set_interior(n, prims[n])
    g.set_interior("W", o.named("W"))
    g.flux_rhs(1)
    for n in RHS_FIELDS:
        assert np.array_equal(g.interior(n, 1), o.named(n, 1), equal_nan=True), n
    g.close()
