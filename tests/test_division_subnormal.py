"""divide_all (cueva_common.cuh) on numerators far below its exponent range,
down to the smallest subnormals: they are no zeros and take the division.

CPU: the range test's key separates zeros from every other value, and the
three operations are not the quotient down there (why the test is needed).
GPU: the stage right-hand side with psi, phi and q of that size equals the
oracle's bit for bit, both spacings being no power of two (with flux routines
4 and 7 also the halves of the HLLC star terms, which round down there).
"""
import ctypes
import ctypes.util

import numpy as np
import pytest

fma = ctypes.CDLL(ctypes.util.find_library("m")).fma
fma.restype = ctypes.c_double
fma.argtypes = [ctypes.c_double] * 3

A_LO = (1023 - 800) << 20


def three_operations(a, b):
    z = 1.0 / b
    q = a * z
    return fma(fma(-b, q, a), z, q)


def takes_the_division(a):
    """magnitude_key and the lower range test of divide_all, in 32-bit words"""
    w = int(np.float64(a).view(np.uint64))
    key = (w >> 32 & 0x7FFFFFFF) | min(w & 0xFFFFFFFF, 1)
    return (key - 1) & 0xFFFFFFFF < A_LO - 1


def test_only_zeros_pass_below_the_range():
    assert not takes_the_division(0.0) and not takes_the_division(-0.0)
    assert not takes_the_division(2.0 ** -800) and not takes_the_division(-1.0)
    for a in [k * 5e-324 for k in (1, 2, 3, 2 ** 31, 2 ** 32 - 1, 2 ** 32)] + [2.0 ** -1022, 2.0 ** -801]:
        assert takes_the_division(a) and takes_the_division(-a), a


def test_three_operations_are_no_quotient_of_subnormals():
    wrong = 0
    for b in (2.0 / 93, 1.0 / 70, 1.3):
        for k in range(1, 2000):
            a = k * 5e-324
            if three_operations(a, b) != a / b:
                assert takes_the_division(a), (a, b)
                wrong += 1
    assert wrong > 0


@pytest.mark.gpu
@pytest.mark.parametrize("solver", [2, 4, 5, 6, 7])
@pytest.mark.parametrize("scale", [1.0e-321, 1.0e-318, 1.0e-314])
def test_stage_rhs_with_subnormal_fields(oracle_mod, solver, scale):
    from cueva import Cueva, RHS_FIELDS, STAGE_FIELDS
    imax, jmax = 45, 37
    kw = dict(order=2, flux_solver=solver, rec_mp=0, c2p=1, bc_x=0, bc_y=1, sigma=1e3)
    g = Cueva(imax, jmax, **kw)
    g.kh_init(v0=0.4, a=0.05)
    rng = np.random.default_rng(11)
    for n in ("psi", "phi", "q"):
        g.set_interior(n, scale * rng.standard_normal((jmax + 1, imax + 1)))
    prims = g.prims()
    oracle_mod.set_libm_seed(0)
    o = oracle_mod.Oracle(imax, jmax, **kw)
    o.set_prims(prims)
    o.run_stages(1)
    for n in STAGE_FIELDS[:17]:
        g.set_interior(n, o.named(n), 1)
    for n in prims:
        g.set_interior(n, prims[n])
    g.set_interior("W", o.named("W"))
    g.flux_rhs(1)
    for n in RHS_FIELDS:
        assert np.array_equal(g.interior(n, 1), o.named(n, 1), equal_nan=True), n
    g.close()
