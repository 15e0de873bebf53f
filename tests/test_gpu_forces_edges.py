"""Forces, face coefficients and right-hand side on grids that end inside, at and next to tile borders, with uniform
gas (corner viscosities taken from the cell) beside varying gas, still and moving: forces within the stated FP32
tolerance of the oracle, coefficients and rhs its bits, every tile shape the same bits."""
import numpy as np
import pytest

import campfire_b200 as cb
from campfire_b200.fluid import load_scene
from conftest import norm_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(15, 17), (33, 7), (40, 64), (64, 16), (72, 88)])
def test_forces_and_rhs_at_edges(oracle_mod, nx, ny):
    sc = cb.generate_scene(0, nx, ny, 0.8, 21)
    rng = np.random.default_rng(nx * ny)
    T = sc["T"].reshape(ny, nx)
    T[:, : nx // 2] = sc["params"]["Tamb"]
    T[:, nx // 2:] = rng.uniform(290, 1900, (ny, nx - nx // 2))
    o = oracle_mod.OracleSim(nx, ny, 0.8, 0.002)
    load_scene(o, sc)
    u2 = rng.uniform(-2, 2, (nx + 1) * ny).astype(np.float32) * (rng.uniform(size=(nx + 1) * ny) < 0.7)
    v2 = rng.uniform(-2, 2, nx * (ny + 1)).astype(np.float32) * (rng.uniform(size=nx * (ny + 1)) < 0.7)
    sq = rng.uniform(-5, 5, 2 * nx * ny).astype(np.float32)
    o.write("U2", u2); o.write("V2", v2); o.write("SQ", sq)
    o.stage("forces")
    uf, vf = o.read("U").astype(np.float32), o.read("V").astype(np.float32)
    o.write("U", uf); o.write("V", vf)
    o.stage("coef_rhs")
    ref = None
    for shape in (0, 1, 2):
        g = cb.FluidSim(0, {"nx": nx, "ny": ny, "dt": 0.002}, width=0.8).init()
        load_scene(g, sc)
        g.set_tiles(0, 0, shape)
        g.writeBuffer("U2", u2); g.writeBuffer("V2", v2); g.writeBuffer("SQ", sq)
        g.run_stage("forces")
        out = {f: g.readBuffer(f) for f in ("U", "V")}
        for f, w in (("U", uf), ("V", vf)):
            assert norm_err(out[f], w) <= 1e-4, (shape, f)
            assert ref is None or np.array_equal(out[f], ref[f]), (shape, f)
            g.writeBuffer(f, w)
        g.run_stage("coef_rhs")
        for l in range(len(g.levels)):
            for f in ("ax", "ay") + (("rhs",) if l == 0 else ()):
                name = f if l == 0 else f"{f}.{l}"
                assert np.array_equal(g.readBuffer(name), o.read(name).astype(np.float32)), (shape, name)
        ref = out
        g.close()
