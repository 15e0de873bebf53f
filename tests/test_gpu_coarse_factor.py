"""The coarsest inverse where its splits can go wrong: coarsest levels of 5 to 32 columns (register windows of 8, 16
and 32 entries, wider than the band or as wide), one and two rounds of columns, several scenes with one window."""
import numpy as np
import pytest

import campfire_b200 as cb
from campfire_b200.fluid import load_scene
from gpu_pairs import make_pair, sync

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(5, 7), (8, 12), (12, 20), (15, 17), (16, 16), (20, 12), (32, 8), (28, 24), (26, 36)])
def test_the_inverse_is_the_oracles_to_the_bit(oracle_mod, nx, ny):
    g, o, _ = make_pair(oracle_mod, nx, ny, kind=0, seed=77 + nx, warm_steps=2, mode=cb.SOLVE_TOL, tol=1e-30, max_cycles=2)
    g.set_coarse_solve(True); o.set_coarse_solve(True)
    g.run_stage("coef_rhs"); o.stage("coef_rhs")
    sync(o, g)
    g.run_stage("pressure"); o.stage("pressure")
    assert np.array_equal(g.readBuffer("p").astype(np.float64), o.read("p"))
    g.close()


@pytest.mark.parametrize("mode", [True, "pipelined"])
def test_scenes_of_several_widths(mode):
    # a scene's pressure does not depend on the widest scene beside it
    dims = [(5, 7), (32, 8), (16, 16), (72, 88)]
    scenes = [cb.generate_scene(0, nx, ny, 0.8, 5 + nx) for nx, ny in dims]
    b = cb.Batch(dims, 0.8, [s["dt"] for s in scenes])
    for v, s in zip(b.scenes, scenes):
        load_scene(v, s)
    b.set_solver(cb.SOLVE_FP64, 1, 1e-30, 4)
    b.set_coarse_solve(mode)
    b.step(3); b.synchronize()
    for (nx, ny), v, s in zip(dims, b.scenes, scenes):
        g = cb.FluidSim(0, {"nx": nx, "ny": ny, "dt": s["dt"]}, width=0.8).init()
        load_scene(g, s)
        g.set_solver(cb.SOLVE_FP64, 1, 1e-30, 4)
        g.set_coarse_solve(mode)
        g.step(3); g.synchronize()
        assert np.array_equal(g.read_p64(), v.read_p64()), (nx, ny)
        g.close()
    b.close()
