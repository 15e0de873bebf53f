"""Advection at the domain's last faces (x = nx, y = ny) where they travel farther than every other site of their tile:
local flow of 2 to 4 cells per step beside the open sides and the top, every tile shape, the oracle's bits."""
import numpy as np
import pytest

import campfire_b200 as cb
from campfire_b200.fluid import load_scene

pytestmark = pytest.mark.gpu


def _bumps(seed, nx, ny, dx, dt):
    """One bump of each velocity component beside the last faces."""
    rng = np.random.default_rng(seed)
    if seed % 2 == 0:
        c0 = np.array([nx - rng.uniform(0, 5), rng.uniform(3, ny - 3)])
    else:
        c0 = np.array([rng.uniform(3, nx - 3), ny - rng.uniform(0, 5)])
    out = []
    for x, y in (np.meshgrid(np.arange(nx + 1.0), np.arange(ny) + 0.5), np.meshgrid(np.arange(nx) + 0.5, np.arange(ny + 1.0))):
        c, s = c0 + rng.uniform(-2, 2, 2), rng.uniform(1, 2.5, 2)
        top = rng.uniform(2, 4) * rng.choice([-1, 1]) * dx / dt
        out.append((top * np.exp(-((x - c[0]) / s[0]) ** 2 - ((y - c[1]) / s[1]) ** 2)).astype(np.float32))
    return out


def _vortex(cx, cy, s, cells, nx, ny, dx, dt):
    """Stream function s exp(-r^2 / s^2), its fastest face at `cells` cells per step."""
    def e(x, y):
        return np.exp(-((y - cy) / s) ** 2 - ((x - cx) / s) ** 2)
    xu, yu = np.meshgrid(np.arange(nx + 1.0), np.arange(ny) + 0.5)
    xv, yv = np.meshgrid(np.arange(nx) + 0.5, np.arange(ny + 1.0))
    U, V = -2 * (yu - cy) / s * e(xu, yu), 2 * (xv - cx) / s * e(xv, yv)
    k = cells * dx / dt / max(np.abs(U).max(), np.abs(V).max())
    return (k * U).astype(np.float32), (k * V).astype(np.float32)


# seeds whose last faces need a ring of first-order values that no other site of their tile needs, by the traces
# evaluated on the host (in some tile shape), then as many that need not
FAR = {(64, 96): (24, 238, 592, 1126, 1298, 1410, 1574, 2232),
       (40, 64): (34, 332, 356, 522, 969, 1126, 1298, 1436, 1516, 2066, 2169, 2232, 2534, 2624),
       (72, 88): (44, 238, 244, 386, 503, 592, 1016, 1058, 1216, 1304, 1436, 1766, 2772, 2953),
       (33, 7): (1386,)}


@pytest.mark.parametrize("nx,ny", sorted(FAR))
def test_last_faces_far_from_their_tile(oracle_mod, nx, ny):
    sc = cb.generate_scene(0, nx, ny, 0.8, 5)
    dx, dt = 0.8 / nx, sc["dt"]
    o = oracle_mod.OracleSim(nx, ny, 0.8, dt)
    load_scene(o, sc)
    sims = []
    for shape in (0, 1, 2):
        g = cb.FluidSim(0, {"nx": nx, "ny": ny, "dt": dt}, width=0.8).init()
        load_scene(g, sc)
        g.set_tiles(shape, 0, 0)
        sims.append(g)
    fields = [_bumps(s, nx, ny, dx, 0.002) for s in FAR[nx, ny] + tuple(range(100))]
    if (nx, ny) == (64, 96):
        fields.append(_vortex(60.5, 41.6, 3.2, -3.6, nx, ny, dx, 0.002))
    for q, (U, V) in enumerate(fields):
        # displacements in cells per step as above, whatever the scene's step
        U, V = (a * np.float32(0.002 / dt) for a in (U, V))
        o.write("U", U.ravel()); o.write("V", V.ravel())
        o.stage("advect")
        for shape, g in enumerate(sims):
            g.writeBuffer("U", U.ravel()); g.writeBuffer("V", V.ravel())
            g.run_stage("advect")
            for f in ("U2", "V2", "T2", "Y2"):
                assert np.array_equal(g.readBuffer(f), o.read(f).astype(np.float32)), (q, shape, f)
    for g in sims:
        g.close()
