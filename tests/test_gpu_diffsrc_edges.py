"""Diffusion + sources on grids that end inside, at and next to tile borders, over the sub-step counts, hot, cold and
fuel-free gas: the oracle within the stated FP32 tolerance (1e-4 of the field's largest value), every tile shape the
same bits, the fixed-point totals to one unit per 8x8 block."""
import numpy as np
import pytest

import campfire_b200 as cb
from campfire_b200.fluid import load_scene
from conftest import norm_err

pytestmark = pytest.mark.gpu
TOL = 1e-4


@pytest.mark.parametrize("nx,ny", [(15, 17), (33, 7), (40, 64), (72, 88)])
@pytest.mark.parametrize("sub", [1, 3, 5])
def test_diffusion_and_sources_at_edges(oracle_mod, nx, ny, sub):
    sc = cb.generate_scene(0, nx, ny, 0.8, 9)
    # hot and burning, cold with fuel, hot without fuel, and gas exactly at rest and ambient, side by side
    rng = np.random.default_rng(nx + sub)
    T, Y = sc["T"].reshape(ny, nx), sc["Y"].reshape(ny, nx, 4)
    q = nx // 4
    T[:, :q] = rng.uniform(1200, 1900, (ny, q))
    Y[:, :q] = np.array([0.05, 0.15, 0.79, 0.01])
    T[:, q:2 * q] = rng.uniform(290, 420, (ny, q))
    Y[:, q:2 * q] = np.array([0.2, 0.18, 0.62, 0.0])
    T[:, 2 * q:3 * q] = rng.uniform(800, 1500, (ny, q))
    Y[:, 2 * q:3 * q] = np.array([0.0, 0.2, 0.795, 0.005])
    T[:, 3 * q:] = sc["params"]["Tamb"]
    Y[:, 3 * q:] = np.array([0.0, sc["params"]["YOamb"], 0.0, 0.0])
    dx = 0.8 / nx
    alpha = 1.716e-5 * (2200 / 273.15) ** 1.5 * 383.55 / (2200 + 110.4) / 0.7 / (101325 * 0.0289 / 8.314462 / 2200)
    dt = (sub - 0.5) * dx * dx / (4.5 * alpha)
    o = oracle_mod.OracleSim(nx, ny, 0.8, dt)
    load_scene(o, sc)
    o.stage("diffuse")
    o.stage("sources")
    acc_o = o.readback()["acc"].astype(np.int64)
    blocks = ((nx + 7) // 8) * ((ny + 7) // 8)
    ref = None
    for shape in (0, 1, 2):
        g = cb.FluidSim(0, {"nx": nx, "ny": ny, "dt": dt}, width=0.8).init()
        load_scene(g, sc)
        assert g.info()["diffSub"] == sub
        g.set_tiles(0, shape, 0)
        g.run_stage("diffuse_sources")
        out = {f: g.readBuffer(f) for f in ("T", "Y", "SQ")}
        acc = g.readback()["acc"].astype(np.int64)
        g.close()
        for f in ("T", "Y", "SQ"):
            assert norm_err(out[f], o.read(f)) <= TOL, (shape, f)
            assert ref is None or np.array_equal(out[f], ref[0][f]), (shape, f)
        # rounding to fixed point per block, and the totals' own relative tolerance
        assert np.all(np.abs(acc[512:514] - acc_o[512:514]) <= blocks + TOL * np.abs(acc_o[512:514]))
        assert abs(acc[514] - acc_o[514]) <= 1 + TOL * abs(acc_o[514])
        assert ref is None or np.array_equal(acc, ref[1])
        ref = (out, acc)
