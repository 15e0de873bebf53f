"""Advection over displacements of a fraction of a cell to beyond the widest staged halo, on grids that end inside,
at and next to tile borders, in every tile shape: the oracle's bits."""
import numpy as np
import pytest

import campfire_b200 as cb
from campfire_b200.fluid import load_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(15, 17), (32, 8), (33, 7), (40, 64), (72, 88), (96, 48)])
@pytest.mark.parametrize("cells", [0.0, 0.4, 1.3, 3.7, 9.0])
def test_advection_bits_over_displacements(oracle_mod, nx, ny, cells):
    sc = cb.generate_scene(0, nx, ny, 0.8, 5)
    rng = np.random.default_rng(nx * 100 + ny)
    top = cells * (0.8 / nx) / sc["dt"]
    # smooth swirls with single fast faces, a quiet half, exact zeros
    for f, w in (("U", nx + 1), ("V", nx)):
        n = sc[f].size // w
        y, x = np.mgrid[0:n, 0:w]
        v = np.sin(0.7 * x + rng.uniform(0, 6)) * np.cos(0.5 * y + rng.uniform(0, 6)) * (x > w // 2)
        v[rng.uniform(size=v.shape) < 0.02] = 1.0
        sc[f] = (top * v).astype(np.float32).ravel()
    o = oracle_mod.OracleSim(nx, ny, 0.8, sc["dt"])
    load_scene(o, sc)
    o.stage("advect")
    for shape in (0, 1, 2):
        g = cb.FluidSim(0, {"nx": nx, "ny": ny, "dt": sc["dt"]}, width=0.8).init()
        load_scene(g, sc)
        g.set_tiles(shape, 0, 0)
        g.run_stage("advect")
        for f in ("T2", "Y2", "U2", "V2"):
            assert np.array_equal(g.readBuffer(f), o.read(f).astype(np.float32)), (shape, f)
        g.close()


@pytest.mark.parametrize("n", [10, 11])
def test_many_tiles_take_the_larger_ones(n):
    # 3840 and 4224 tiles of 32x8 cells: the default shape on either side of its line gives shape 0's bits
    out = []
    for explicit in (False, True):
        b = cb.Batch([(256, 384)] * n, 0.8, [0.002] * n)
        for k in (0, n - 1):
            load_scene(b.scenes[k], cb.generate_scene(0, 256, 384, 0.8, 3 + k))
        if explicit:
            b.set_tiles(0, 0, 0)
        b.step(1); b.synchronize()
        out.append([b.scenes[k].readBuffer(f) for k in (0, n - 1) for f in ("T", "Y", "U", "V")])
        b.close()
    assert all(np.array_equal(x, y) for x, y in zip(*out))
