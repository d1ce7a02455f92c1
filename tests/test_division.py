"""The shared-divisor division of the kernels (divide_all, cueva_common.cuh).

CPU: its three operations give the correctly rounded quotient, on random
operands and on quotients within 2^-50 ulp of a rounding boundary.  GPU: the
stage right-hand side, whose flux differences are divided that way where the
spacing is no power of two, equals the oracle's bit for bit when fields are
zero, far below the tested exponent range and far above it.
"""
import ctypes
import ctypes.util

import numpy as np
import pytest

fma = ctypes.CDLL(ctypes.util.find_library("m")).fma
fma.restype = ctypes.c_double
fma.argtypes = [ctypes.c_double] * 3


def quotient(a, b):
    z = 1.0 / b
    q = a * z
    return fma(fma(-b, q, a), z, q)


def hard_numerators(b, rng, count):
    """Numerators a (53-bit significands) with a / b close to the midpoint of
    two doubles: for b = m 2^e, integers A with 2^54 A = (2k + 1) m + d and
    |d| small, solved for A modulo m."""
    m = int(np.ldexp(np.frexp(b)[0], 53))
    if m % 2 == 0:
        m += 1
    out = []
    inv = pow(1 << 54, -1, m)
    for d in range(1, 4 * count):
        for s in (d, -d):
            A = (s * inv) % m
            if A >= 1 << 52 and (((A << 54) - s) // m) % 2 == 1:
                out.append(float(A))
    return float(m), out[:count]


def test_three_operation_quotient_is_correctly_rounded():
    rng = np.random.default_rng(7)
    worst = 0
    for b in (2.0 / 93, 1.0 / 70, 2.0 / 1003, 1.0 / 611, 2.0 / 4093, 0.999, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52,
              1.0e-3, 1.9990000000000001):
        for a in rng.standard_normal(20000) * 10.0 ** rng.uniform(-30, 30, 20000):
            worst += quotient(float(a), b) != float(a) / b
        m, hard = hard_numerators(b, rng, 2000)
        for a in hard:
            worst += quotient(a, m) != a / m
    assert worst == 0


@pytest.mark.gpu
@pytest.mark.parametrize("solver", [2, 5, 6, 7])
@pytest.mark.parametrize("scale", [0.0, 1.0e-290, 1.0e-200, 1.0, 1.0e250])
def test_stage_rhs_with_extreme_fields(oracle_mod, solver, scale):
    """psi, phi and q scaled to zero, below and above the tested exponents;
    both spacings are no power of two."""
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
