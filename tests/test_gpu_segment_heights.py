"""Segment heights of the fused stage kernel's tiles (stage_seg_rows), read
from the grid of its launches: strips of 31 points by segments of 8 nb - 1
rows, nb being the count measured fastest or within the noise of it."""
import json
import time

import pytest

pytestmark = pytest.mark.gpu


def launched_tiles(path, run):
    """CTAs of each k_stage launch of run()"""
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        time.sleep(0.005)   # the launches well inside the recorded window
        run()
        time.sleep(0.005)
    prof.export_chrome_trace(path)
    with open(path) as f:
        ev = json.load(f)["traceEvents"]
    return [e["args"]["grid"][0] for e in ev if "k_stage" in e.get("name", "") and "grid" in e.get("args", {})]


def tiles(imax, jmax, nb):
    return ((imax + 31) // 31) * ((jmax + 8 * nb - 1) // (8 * nb - 1))


@pytest.mark.parametrize("imax,jmax,solver,bands", [
    (200, 200, 2, 1), (300, 300, 4, 2), (300, 300, 1, 2), (400, 300, 2, 2), (512, 256, 1, 2),   # MC slopes, few waves
    (500, 500, 2, 2), (1000, 500, 2, 2), (1000, 1000, 4, 3),
    (300, 300, 7, 1), (500, 500, 7, 2), (500, 500, 6, 2), (900, 900, 7, 3), (1000, 1000, 5, 3), (1000, 500, 7, 2)])
def test_single_grids(tmp_path, imax, jmax, solver, bands):
    from cueva import Cueva
    g = Cueva(imax, jmax, order=2, flux_solver=solver, sigma=1e3)
    g.kh_init(v0=0.5, a=0.05)
    g.upload()
    g.sync()

    def run():
        g.profile_steps(1)   # one launch per stage, each waited for

    assert launched_tiles(str(tmp_path / "t.json"), run) == [tiles(imax, jmax, bands)] * 2
    g.close()
