"""The pressure stage's bits over level shapes: the coarsest level's 120 red-black sweeps in one warp's registers
(and the wider and taller levels that keep the block's passes), and the tiled smoothers on levels whose widths
and heights end inside a tile, a thread's four cells or a coarse pair."""
import numpy as np
import pytest

import campfire_b200 as cb
from campfire_b200.fluid import load_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(2, 128), (3, 85), (7, 36), (8, 12), (10, 14), (11, 23), (15, 17), (16, 16), (31, 8),
                                   (32, 8), (17, 15), (22, 11), (33, 7), (64, 4), (128, 2), (2, 2), (5, 3),
                                   (22, 46), (56, 80)])
def test_sweeps_bits_over_coarsest_shapes(oracle_mod, nx, ny):
    _same_pressure(oracle_mod, nx, ny, 6144)


@pytest.mark.parametrize("nx,ny", [(32, 16), (34, 18), (36, 48), (44, 60), (72, 88), (104, 136), (176, 208), (18, 56)])
def test_tiled_levels_bits_over_shapes(oracle_mod, nx, ny):
    _same_pressure(oracle_mod, nx, ny, 1)   # every level but the coarsest tiled


def _same_pressure(oracle_mod, nx, ny, cells):
    sc = cb.generate_scene(0, nx, ny, 0.8, 77)
    # pieces of a few cells, so that closed cells and partly open faces occur on the coarsest level too
    sc["pieces"][3::20][: sc["npieces"]] = 0.08
    g = cb.FluidSim(0, {"nx": nx, "ny": ny, "dt": sc["dt"]}, width=0.8).init()
    o = oracle_mod.OracleSim(nx, ny, 0.8, sc["dt"])
    for s in (g, o):
        load_scene(s, sc)
        s.set_solver(cb.SOLVE_FIXED, 2)
    g.set_coarse_cells(cells)
    o.stage("coef_rhs")
    for f in ("ax", "ay", "rhs"):
        for lvl in range(len(g.levels)):
            name = f if lvl == 0 else f"{f}.{lvl}"
            if f != "rhs" or lvl == 0:
                g.writeBuffer(name, o.read(name))
    g.run_stage("pressure"); o.stage("pressure")
    a, b = g.readBuffer("p"), o.read("p").astype(np.float32)
    g.close()
    assert np.abs(b).max() > 0
    assert np.array_equal(a, b)
