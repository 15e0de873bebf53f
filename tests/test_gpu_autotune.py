"""The autotuner times schedules that an engine runs: every candidate a schedule of its own, the chosen one as timed."""
import pytest

import campfire_b200 as cb
from campfire_b200.fluid import load_scene

pytestmark = pytest.mark.gpu


def _launches(nx, ny, cells, fp64):
    sc = cb.generate_scene(0, nx, ny, 0.8, 7)
    g = cb.FluidSim(0, {"nx": nx, "ny": ny, "dt": sc["dt"]}, width=0.8).init()
    load_scene(g, sc)
    if fp64:
        g.set_solver(cb.SOLVE_FP64, 1, 1e-6, 1)
        g.set_coarse_solve(True)
    else:
        g.set_solver(cb.SOLVE_FIXED, 1)
    g.set_coarse_cells(cells)
    g.step(1)
    g.synchronize()
    n = g.launch_count()
    g.close()
    return n


@pytest.mark.parametrize("nx,ny", [(256, 384), (112, 160), (32, 48), (15, 17)])
@pytest.mark.parametrize("fp64", [False, True])
def test_candidates_are_schedules_of_their_own(nx, ny, fp64):
    if (nx, ny) == (15, 17):
        # one level only: nothing to choose
        with pytest.raises(cb.CampfireError):
            cb.autotune([(nx, ny)], iters=2, coarse_direct=fp64)
        return
    r = cb.autotune([(nx, ny)], iters=2, coarse_direct=fp64)
    cells = sorted(r["ms_per_cycle"])
    assert r["best"] in cells and r["ms_per_cycle"][r["best"]] == min(r["ms_per_cycle"].values())
    # a block that starts one level earlier saves that level's two launches per cycle
    n = [_launches(nx, ny, c, fp64) for c in cells]
    assert all(a - b >= 2 for a, b in zip(n, n[1:])), dict(zip(cells, n))
    # the largest candidate stands for every larger request, level 0 aside
    assert _launches(nx, ny, nx * ny - 1, fp64) == n[-1]


def test_candidates_of_an_uneven_batch():
    r = cb.autotune([(96, 144), (256, 384), (128, 192)], iters=2, coarse_direct=True)
    # the levels of at most 2048 cells, and the one request that starts every block at the largest of them
    assert max(r["ms_per_cycle"]) <= 2048 and len(r["ms_per_cycle"]) >= 3
