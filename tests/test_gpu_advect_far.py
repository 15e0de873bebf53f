"""Advection from trace points millions of cells away: the boundary values that the oracle reads there, its bits."""
import numpy as np
import pytest

import campfire_b200 as cb
from campfire_b200.fluid import load_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [1e5, 5e6, 1.8e7, 1e9])
def test_advection_from_points_millions_of_cells_away(oracle_mod, cells):
    nx, ny = 40, 64
    sc = cb.generate_scene(0, nx, ny, 0.8, 9)
    rng = np.random.default_rng(3)
    speed = cells * (0.8 / nx) / sc["dt"]
    for f in ("U", "V"):
        v = sc[f].copy()
        at = rng.uniform(size=v.size) < 0.03
        v[at] = (speed * rng.choice([-1.0, 1.0], at.sum())).astype(np.float32)
        sc[f] = v
    o = oracle_mod.OracleSim(nx, ny, 0.8, sc["dt"])
    load_scene(o, sc)
    o.stage("advect")
    for shape in (0, 1, 2):
        g = cb.FluidSim(0, {"nx": nx, "ny": ny, "dt": sc["dt"]}, width=0.8).init()
        load_scene(g, sc)
        g.set_tiles(shape, 0, 0)
        g.run_stage("advect")
        for f in ("T2", "Y2", "U2", "V2"):
            assert np.array_equal(g.readBuffer(f), o.read(f).astype(np.float32), equal_nan=True), (shape, f)
        g.close()
