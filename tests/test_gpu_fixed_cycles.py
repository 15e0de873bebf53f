"""Cycles laid out in the step graph (up to twelve) and looped there, against kernel-by-kernel launches, and the
coarse block's start asked for at different sizes: the same bits; the FP64 modes keep a block over level 0."""
import numpy as np
import pytest

import campfire_b200 as cb
from campfire_b200.fluid import load_scene

pytestmark = pytest.mark.gpu
FIELDS = ("T", "Y", "U", "V", "p")


def _run(nx, ny, ncycles, graphs, cells, steps=3):
    sc = cb.generate_scene(2, nx, ny, 0.8, 41)
    g = cb.FluidSim(0, {"nx": nx, "ny": ny, "dt": sc["dt"]}, width=0.8).init()
    load_scene(g, sc)
    g.set_solver(cb.SOLVE_FIXED, ncycles)
    g.set_graphs(graphs)
    g.set_coarse_cells(cells)
    g.step(steps)
    g.synchronize()
    out = {f: g.readBuffer(f) for f in FIELDS}
    inf = g.info()
    g.close()
    return out, inf


@pytest.mark.parametrize("nx,ny", [(15, 17), (32, 48), (64, 96), (112, 160)])
@pytest.mark.parametrize("ncycles", [1, 2, 12, 13])
def test_unrolled_cycles_equal_launched_ones(nx, ny, ncycles):
    ref, inf = _run(nx, ny, ncycles, False, 1536)
    assert inf["last_cycles"] == ncycles
    for graphs, cells in ((True, 1536), (True, 6144), (True, 100000), (False, 6144)):
        out, i2 = _run(nx, ny, ncycles, graphs, cells)
        assert i2["last_cycles"] == ncycles
        for f in FIELDS:
            assert np.array_equal(out[f], ref[f]), (graphs, cells, f)


@pytest.mark.parametrize("mode,tol,krylov", [(cb.SOLVE_TOL, 0.3, 0), (cb.SOLVE_TOL, 1e-5, 0), (cb.SOLVE_FP64, 1e-2, 1),
                                             (cb.SOLVE_FP64, 1e-6, 1), (cb.SOLVE_FP64, 1e-13, 1),
                                             (cb.SOLVE_FP64, 1e-8, 3), (cb.SOLVE_FP64, 1e-9, 0)])
def test_cycles_to_a_tolerance_equal_launched_ones(mode, tol, krylov):
    # fewer cycles than are laid out, as many, and more (the loop's share)
    sc = cb.generate_scene(0, 128, 192, 0.8, 44)
    res = []
    for graphs in (True, False):
        g = cb.FluidSim(0, {"nx": 128, "ny": 192, "dt": sc["dt"]}, width=0.8).init()
        load_scene(g, sc)
        g.set_solver(mode, 1, tol, 40)
        g.set_krylov(krylov)
        g.set_graphs(graphs)
        cyc = []
        for _ in range(4):
            g.step(1)
            cyc.append(g.info()["last_cycles"])
        res.append((cyc, {f: g.readBuffer(f) for f in FIELDS}, g.read_p64()))
        g.close()
    assert res[0][0] == res[1][0]
    for f in FIELDS:
        assert np.array_equal(res[0][1][f], res[1][1][f]), f
    assert np.array_equal(res[0][2], res[1][2])


def test_unrolled_cycles_in_a_batch():
    dims = [(64, 96), (32, 48), (96, 144)]
    scenes = [cb.generate_scene(2, nx, ny, 0.8, 50 + k) for k, (nx, ny) in enumerate(dims)]
    res = []
    for graphs in (True, False):
        b = cb.Batch(dims, 0.8, [s["dt"] for s in scenes])
        for v, s in zip(b.scenes, scenes):
            load_scene(v, s)
        b.set_solver(cb.SOLVE_FIXED, 2)
        b.set_graphs(graphs)
        b.step(3)
        b.synchronize()
        res.append([cb.field_hash(v) for v in b.scenes])
        b.close()
    assert res[0] == res[1]


def test_solver_changes_move_the_block():
    # 64x96 = 6144 cells: the FP64 modes run its whole hierarchy in the block when asked to (the update kernel
    # follows), fixed cycles do not; results after going there and back are those of never having gone
    sc = cb.generate_scene(2, 64, 96, 0.8, 43)

    def run(switch):
        g = cb.FluidSim(0, {"nx": 64, "ny": 96, "dt": sc["dt"]}, width=0.8).init()
        load_scene(g, sc)
        if switch:
            g.set_solver(cb.SOLVE_FP64, 1, 1e-6, 50)
            g.set_krylov(True)
            assert not g.krylov_folded()
            g.set_coarse_cells(1536)
            assert g.krylov_folded()
            g.set_coarse_cells(6144)
            assert not g.krylov_folded()
        g.set_solver(cb.SOLVE_FIXED, 2)
        g.step(2)
        h = cb.field_hash(g)
        g.close()
        return h

    assert run(False) == run(True)
