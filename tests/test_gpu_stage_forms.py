"""Every form of the fused stage kernel against the two kernels, bit for bit,
with the form that ran read from the block and grid of its launches: the wide
form at each of its heights of 4 to 12 warps (up to 148 tiles), and the ring
with several bands per tile, with stored right-hand sides and both stage-sum
modes (orders 3 and 4), copy and periodic x, FP64 and mixed precision."""
import json
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def state(imax, jmax):
    from cueva import PRIM_FIELDS
    rng = np.random.default_rng(imax * 1000 + jmax)
    y, x = np.meshgrid(np.linspace(0, 1, jmax + 1), np.linspace(-1, 1, imax + 1), indexing="ij")
    out = {}
    for n in PRIM_FIELDS:
        w = sum(rng.uniform(0.3, 1) * np.sin(2 * np.pi * m * y + rng.uniform(0, 6)) * np.cos(np.pi * m * x + 1)
                for m in (1, 2, 5))
        out[n] = (1.0 if n in ("rho", "p") else 0.0) + 0.03 * w
    out["vy"] = out["vy"] + 0.4 * np.tanh(x / 0.05)
    return out


def run(kw, two_kernels, path):
    """state after two steps, and (warps, CTAs) of the k_stage launches of a third"""
    from torch.profiler import ProfilerActivity, profile

    from cueva import Cueva
    g = Cueva(**kw)
    if two_kernels:
        g.set_stage_kernel(0)
    for n, a in state(kw["imax"], kw["jmax"]).items():
        g.set_interior(n, a)
    g.upload()
    g.step(2)
    g.download()
    out = {n: g.interior(n).copy() for n in state(8, 8)}
    shapes = set()
    if not two_kernels:
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            time.sleep(0.005)   # the launches well inside the recorded window
            g.profile_steps(1)
            time.sleep(0.005)
        prof.export_chrome_trace(path)
        with open(path) as f:
            for e in json.load(f)["traceEvents"]:
                if "k_stage" in e.get("name", "") and "grid" in e.get("args", {}):
                    shapes.add((e["args"]["block"][1], e["args"]["grid"][0]))
    g.close()
    return out, shapes


def compare(kw, tmp_path):
    a, shapes = run(kw, False, str(tmp_path / "t.json"))
    b, _ = run(kw, True, None)
    for n in a:
        assert np.array_equal(a[n], b[n]), n
    assert len(shapes) == 1
    return shapes.pop()


@pytest.mark.parametrize("imax,jmax,warps", [(6, 6, 4), (122, 109, 4), (122, 146, 5), (200, 100, 6), (122, 220, 7),
                                             (155, 145, 8), (122, 294, 9), (256, 128, 10), (215, 208, 11),
                                             (215, 229, 12), (279, 140, 12)])
@pytest.mark.parametrize("solver,rec,precision", [(5, 0, 0), (6, 0, 0), (7, 0, 0), (7, 0, 1), (6, 1, 1), (7, 1, 0),
                                                  (5, 2, 0), (7, 2, 1)])
def test_wide_heights(tmp_path, imax, jmax, warps, solver, rec, precision):
    kw = dict(imax=imax, jmax=jmax, order=4, intsum_reset=1, flux_solver=solver, rec_mp=rec, precision=precision,
              sigma=1e3, bc_x=imax % 2)
    shape = compare(kw, tmp_path)
    assert shape == (warps, ((imax + 31) // 31) * ((jmax + warps - 1) // (warps - 1))) and shape[1] <= 148


@pytest.mark.parametrize("imax,jmax", [(500, 500), (611, 1003)])
@pytest.mark.parametrize("solver,order,reset,precision,bc_x", [(7, 4, 1, 0, 0), (7, 4, 0, 1, 1), (5, 4, 1, 0, 1),
                                                               (6, 3, 0, 0, 1), (6, 4, 1, 1, 0), (2, 4, 1, 0, 1),
                                                               (4, 3, 1, 0, 0), (1, 4, 0, 0, 0), (3, 4, 1, 0, 1),
                                                               (4, 4, 1, 1, 1)])
def test_ring_of_several_bands(tmp_path, imax, jmax, solver, order, reset, precision, bc_x):
    kw = dict(imax=imax, jmax=jmax, order=order, intsum_reset=reset, flux_solver=solver, rec_mp=0,
              precision=precision, sigma=1e3, bc_x=bc_x)
    warps, ctas = compare(kw, tmp_path)
    assert warps == 8 and ctas < ((imax + 31) // 31) * ((jmax + 7) // 7)
