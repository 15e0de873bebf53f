"""A temperature that is not a number spreads through open faces, as in the oracle: a diverged run shows."""
import numpy as np
import pytest

import campfire_b200 as cb
from campfire_b200.fluid import load_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sub", [1, 3])
def test_diffusion_spreads_a_temperature_that_is_not_a_number(oracle_mod, sub):
    nx, ny = 40, 64
    sc = cb.generate_scene(0, nx, ny, 0.8, 9)
    T = sc["T"].reshape(ny, nx)
    for i, j in ((0, 0), (7, 30), (8, 30), (31, 15), (32, 16), (39, 63)):
        T[j, i] = np.nan
    dx = 0.8 / nx
    alpha = 1.716e-5 * (2200 / 273.15) ** 1.5 * 383.55 / (2200 + 110.4) / 0.7 / (101325 * 0.0289 / 8.314462 / 2200)
    dt = (sub - 0.5) * dx * dx / (4.5 * alpha)
    o = oracle_mod.OracleSim(nx, ny, 0.8, dt)
    load_scene(o, sc)
    o.stage("diffuse")
    want = o.read("T")
    assert np.isnan(want).sum() > 6
    for shape in (0, 1, 2):
        g = cb.FluidSim(0, {"nx": nx, "ny": ny, "dt": dt}, width=0.8).init()
        load_scene(g, sc)
        assert g.info()["diffSub"] == sub
        g.set_tiles(0, shape, 0)
        g.run_stage("diffuse")
        got = g.readBuffer("T")
        g.close()
        assert np.array_equal(np.isnan(got), np.isnan(want)), shape
        ok = ~np.isnan(want)
        # the FP32 tolerance of the diffusion tests
        assert np.max(np.abs(got[ok] - want[ok])) <= 1e-4 * np.max(np.abs(want[ok])), shape
