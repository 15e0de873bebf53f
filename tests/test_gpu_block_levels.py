"""The one-CTA coarse block over levels of more than 2048 cells, where an engine still runs them there: level 0 whole
in the FP64 modes, the W tail's level. Against the tiled kernels' bits and the oracle."""
import numpy as np
import pytest

import campfire_b200 as cb
from campfire_b200.fluid import load_scene
from conftest import norm_err

pytestmark = pytest.mark.gpu


def _sim(nx, ny, cells, krylov=0, w=0):
    sc = cb.generate_scene(1, nx, ny, 0.8, 77)
    g = cb.FluidSim(0, {"nx": nx, "ny": ny, "dt": sc["dt"]}, width=0.8).init()
    load_scene(g, sc)
    g.set_solver(cb.SOLVE_FP64, 1, 1e-10, 300)
    g.set_coarse_solve("pipelined" if w else True)
    g.set_krylov(krylov)
    g.set_coarse_cells(cells)
    g.set_coarse_w(w)
    return g, sc


@pytest.mark.parametrize("nx,ny", [(64, 96), (48, 80), (56, 80)])
def test_block_over_level_0_equals_tiles(nx, ny):
    out = []
    for cells in (6144, 384):
        g, _ = _sim(nx, ny, cells)
        g.step(3)
        g.synchronize()
        out.append((g.info()["last_cycles"], g.launch_count(), g.read_p64(), [g.readBuffer(f) for f in ("T", "Y", "U", "V", "p")]))
        g.close()
    assert out[0][0] == out[1][0] and out[0][1] < out[1][1]
    assert np.array_equal(out[0][2], out[1][2])
    assert all(np.array_equal(a, b) for a, b in zip(out[0][3], out[1][3]))


def test_w_tail_over_3840_cells_matches_the_oracle(oracle_mod):
    # 48x80 cells two levels above the coarsest (12x20) of 192x320; the bounds of the W tail's other parity test
    nx, ny = 192, 320
    g, sc = _sim(nx, ny, 1536, krylov=1, w=4096)
    v, _ = _sim(nx, ny, 1536, krylov=1, w=0)
    for s in (g, v):
        s.step(3)
        s.synchronize()
    # per cycle the block's level saves two tiled launches against the V-cycle's schedule
    per = [(s.launch_count() / s.info()["last_cycles"]) for s in (g, v)]
    assert per[0] < per[1]
    v.close()
    o = oracle_mod.OracleSim(nx, ny, 0.8, sc["dt"])
    load_scene(o, sc)
    o.set_solver(cb.SOLVE_FP64, 1, 1e-10, 300)
    o.set_coarse_solve("pipelined")
    o.set_krylov(True)
    o.set_coarse_w(4096)
    o.copy_state_from(g)
    for k in range(2):
        g.step(1)
        o.step(1)
        gi, oi = g.info(), o.info()
        assert gi["last_rel"] <= 1e-10 and oi["last_rel"] <= 1e-10, k
        assert abs(gi["last_cycles"] - oi["last_cycles"]) <= 2, (k, gi["last_cycles"], oi["last_cycles"])
        for f in ("T", "Y", "U", "V"):
            assert norm_err(g.readBuffer(f), o.read(f)) <= 1e-4, (k, f)
        assert norm_err(g.read_p64(), o.read("p64")) <= 1e-4
    g.close()
