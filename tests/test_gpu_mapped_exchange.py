"""Small pinned exchanges in one launch (k_upload_begin, k_download): the same
state and stage-1 preparation as the copy-engine path, on grids on both sides
of the size limit, and the copy path wherever one of the 14 arrays cannot be
reached by the kernels (not pinned, or not 8-byte aligned)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fields(imax, jmax):
    from cueva import PRIM_FIELDS
    rng = np.random.default_rng(imax)
    shape = (jmax + 13, imax + 13)
    out = {n: 0.01 * rng.standard_normal(shape) for n in PRIM_FIELDS}
    for n in ("rho", "p"):
        out[n] += 1.0
    return out


def bind(g, name, addr):
    from cueva import FIELDS
    assert g.L.cueva_bind_field(g.ctx, FIELDS.index(name), ctypes.cast(addr, ctypes.POINTER(ctypes.c_double))) == 0


def exchange(g, ghost_check=True):
    from cueva import G_CONS, G_PRIMS
    g.upload()
    g.step(1)
    g.download()
    a = {n: g.arrays[n].copy() for n in fields(8, 8)}
    g.download(G_PRIMS | G_CONS)   # always the copy path
    for n in a:
        assert np.array_equal(a[n], g.arrays[n]), n
    for n in ("D", "tau", "Sx", "Sy", "Sz", "W"):
        a[n] = g.interior(n).copy()
    return a


@pytest.mark.parametrize("imax,jmax", [(6, 6), (31, 8), (64, 32), (255, 127), (330, 280), (331, 285)])
def test_mapped_equals_copied(imax, jmax):
    from cueva import Cueva
    init = fields(imax, jmax)
    got = []
    for pinned in (True, False):
        g = Cueva(imax, jmax, order=2, flux_solver=5, sigma=1e3, pinned=pinned)
        for n, a in init.items():
            g.arrays[n][...] = a
        got.append(exchange(g))
        g.close()
    for n in got[0]:
        assert np.array_equal(got[0][n], got[1][n]), n
    for n, a in init.items():   # ghosts are the caller's
        for edge in (np.s_[:6, :], np.s_[-6:, :], np.s_[:, :6], np.s_[:, -6:]):
            assert np.array_equal(got[0][n][edge], a[edge]), n


@pytest.mark.parametrize("case", ["one not pinned", "misaligned"])
def test_unreachable_arrays_take_the_copy_path(case):
    from cueva import Cueva
    imax, jmax = 40, 24
    init = fields(imax, jmax)
    ref = Cueva(imax, jmax, order=2, flux_solver=5, sigma=1e3)
    g = Cueva(imax, jmax, order=2, flux_solver=5, sigma=1e3, pinned=True)
    for h in (ref, g):
        for n, a in init.items():
            h.arrays[n][...] = a
    keep = np.zeros(init["vx"].nbytes + 16, dtype=np.uint8)
    if case == "misaligned":   # pinned, 4 bytes off a double
        assert g.L.cueva_pin_host(keep.ctypes.data_as(ctypes.c_void_p), keep.nbytes) == 0
        addr = (keep.ctypes.data + 7) // 8 * 8 + 4
    else:
        addr = (keep.ctypes.data + 7) // 8 * 8
    ctypes.memmove(addr, init["vx"].ctypes.data, init["vx"].nbytes)
    bind(g, "vx", addr)
    for h in (ref, g):
        h.upload()
        h.step(1)
        h.download()
    back = np.empty_like(init["vx"])
    ctypes.memmove(back.ctypes.data, addr, back.nbytes)
    assert np.array_equal(back, ref.arrays["vx"])
    for n in init:
        if n != "vx":
            assert np.array_equal(g.arrays[n], ref.arrays[n]), n
    g.close()
    ref.close()
    if case == "misaligned":
        g.L.cueva_unpin_host(keep.ctypes.data_as(ctypes.c_void_p))


def test_status_of_a_failed_step_comes_with_the_mapped_download():
    from cueva import CUEVA_ERR_PHYSICS, Cueva, CuevaError
    g = Cueva(32, 16, order=2, flux_solver=5, sigma=1e3, pinned=True)
    for n, a in fields(32, 16).items():
        g.arrays[n][...] = a
    g.arrays["p"][...] = np.nan
    g.upload()
    g.step(1)
    with pytest.raises(CuevaError) as e:
        g.download()
    assert e.value.code == CUEVA_ERR_PHYSICS
    g.clear_status()
    g.close()
