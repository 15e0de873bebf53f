"""The passes beside the gas step at the sizes where their work splits can go wrong: radiation over ray and
piece counts (ray tiles of 64, lanes sharing the pieces), geometry with many pieces (per-tile piece lists),
the renderer's persistent tiles, and the FP64 sums over one to many CTAs."""
import math

import numpy as np
import pytest

import campfire_b200 as cb
from campfire_b200.fluid import load_scene
from campfire_b200.render import Renderer, render_device
from conftest import norm_err

pytestmark = pytest.mark.gpu


def _scene(nx, ny, npieces, seed):
    """A generated scene's gas with `npieces` rotated squares of its own, some touching or beyond the domain."""
    sc = cb.generate_scene(0, nx, ny, 0.8, seed)
    rng = np.random.default_rng(seed)
    a = np.zeros((64, 20), np.float32)
    H = 0.8 / nx * ny
    for n in range(npieces):
        a[n] = [rng.uniform(-0.05, 0.85), rng.uniform(0.0, H), rng.uniform(-3, 3), rng.uniform(0.005, 0.03), 0, 0, 0,
                0.0 if n % 7 == 5 else 1.0, *rng.uniform(400, 1000, 4), *([0.0] * 8)]
    sc.update(pieces=a.ravel(), npieces=npieces)
    return sc


def _pair(oracle_mod, nx, ny, npieces, seed):
    sc = _scene(nx, ny, npieces, seed)
    g = cb.FluidSim(0, {"nx": nx, "ny": ny, "dt": sc["dt"]}, width=0.8).init()
    o = oracle_mod.OracleSim(nx, ny, 0.8, sc["dt"])
    for s in (g, o):
        load_scene(s, sc)
    return g, o


@pytest.mark.parametrize("nx,ny,npieces,nray", [(32, 48, 0, 1), (32, 48, 1, 2), (36, 48, 3, 16), (40, 64, 17, 32),
                                                (96, 144, 33, 64), (64, 96, 64, 128), (15, 17, 2, 1024)])
def test_radiation_over_rays_and_pieces(oracle_mod, nx, ny, npieces, nray):
    g, o = _pair(oracle_mod, nx, ny, npieces, 31 + nray)
    for s in (g, o):
        s.set_nray(nray)
    g.setFrame(5); o.set_frame(5)
    g.writeParams(); o.write_params()
    # twice: the second pass blends into the first's result
    for _ in range(2):
        g.encodeRadiation(); o.radiation()
    rg, ro = g.readback()["rad"].reshape(-1, 4), o.readback()["rad"].reshape(-1, 4)
    g.close()
    # device and host sine and cosine differ by an ulp: a ray moves by ~1e-7 m, which can shift a sample into the
    # next cell (one of a target's samples) and very rarely a grazing ray past a corner
    for k in (0, 1):
        scale = max(float(np.abs(ro[:, k]).max()), 1e-30)
        err = np.abs(rg[:, k].astype(np.float64) - ro[:, k]) / scale
        assert np.mean(err > 1e-3) <= 0.02 and np.median(err) <= 1e-5, (k, err.max())


@pytest.mark.parametrize("nx,ny,npieces", [(15, 17, 0), (32, 48, 1), (72, 88, 33), (224, 320, 64)])
def test_geometry_with_many_pieces(oracle_mod, nx, ny, npieces):
    g, o = _pair(oracle_mod, nx, ny, npieces, 7)
    for f in ("fx", "fy"):
        # rotated pieces: an ulp of the sine and cosine at a distance of ~1 m, in units of a cell
        assert np.abs(g.readBuffer(f) - o.read(f)).max() <= 1e-5 * max(1.0, nx / 32), f
    cg, co = g.readBuffer("cellG").reshape(-1, 2), o.read("cellG").reshape(-1, 2)
    assert norm_err(cg[:, 0], co[:, 0]) <= 1e-6
    # cells on the border between two pieces or faces may go to either
    assert np.mean(cg[:, 1].view(np.uint32) == co[:, 1].astype(np.uint32)) >= 0.995
    g.close()


def _image(sim, W, H, view):
    import torch
    ren = Renderer(sim)
    rng = np.random.default_rng(3)
    w = rng.uniform(0.001, 1.0, (64, 12)).astype(np.float32)
    w[:, 0:4] *= 800
    ren.writeWood(w)
    ren.writeParams({"view": view, "exposure": 1.0, "time": 0.0})
    img = torch.empty(H, W, 4, device="cuda")
    render_device(sim, ren.rp, W, H, img.data_ptr(), ren.wood)
    sim.synchronize()
    return img.cpu().numpy()


@pytest.mark.parametrize("view", ["photo", "temperature"])
@pytest.mark.parametrize("W,H,npieces", [(1, 1, 1), (16, 33, 0), (47, 50, 40), (480, 497, 64)])
def test_a_pixel_does_not_depend_on_its_image(view, W, H, npieces):
    # the centre of pixel (x, y) is the centre of pixel (3x+1, 3y+1) of an image three times as large, to the bit
    # (both are one correctly rounded quotient of the same number); 1440x1491 is several rounds of the CTAs
    sc = _scene(64, 96, npieces, 11)
    g = cb.FluidSim(0, {"nx": 64, "ny": 96, "dt": sc["dt"]}, width=0.8).init()
    load_scene(g, sc)
    g.step(2)
    small, big = _image(g, W, H, view), _image(g, 3 * W, 3 * H, view)
    g.close()
    assert np.array_equal(small.view(np.uint32), big[1::3, 1::3].copy().view(np.uint32))


@pytest.mark.parametrize("nx,ny", [(2, 2), (15, 17), (16, 32), (224, 320), (512, 768)])
def test_monitor_sums(oracle_mod, nx, ny):
    g, o = _pair(oracle_mod, nx, ny, 3, 5)
    g.step(1)
    T, Y = g.readBuffer("T").astype(np.float64), g.readBuffer("Y").astype(np.float64).reshape(-1, 4)
    G, SQ = g.readBuffer("cellG").reshape(-1, 2), g.readBuffer("SQ").astype(np.float64).reshape(-1, 2)
    gas = ~((G[:, 0] < 0) & (G[:, 1].view(np.uint32) != 0xffffffff))
    p = g.params
    dx2 = float(np.float32(p["dx"])) ** 2
    m = p["rhoAmb"] * p["Tamb"] / T[gas] * dx2
    total = lambda v: math.fsum(v.tolist())   # noqa: E731  (correctly rounded)
    want = [total(m), total(m * p["cp"] * T[gas]), *(total(m * Y[gas, k]) for k in range(4)),
            total(SQ[gas, 1]) * dx2, T[gas].max()]
    # the same terms added in another order, in FP64: partial sums of at most ~1e3 terms of one sign
    assert np.allclose(g.budgets(), want, rtol=1e-12, atol=1e-300)
    assert np.array_equal(g.budgets(), g.budgets())
    o.copy_state_from(g)
    a, b = g.pressure_residual(), o.pressure_residual()
    assert abs(a - b) <= 1e-9 * max(abs(b), 1e-12)
    g.close()


@pytest.mark.parametrize("npieces,nray", [(0, 256), (1, 128), (5, 64), (3, 8)])
def test_radiation_rays_shared_by_a_cluster(oracle_mod, npieces, nray):
    # few targets: 16 rays per CTA, one to eight CTAs a target, one or two rounds each
    test_radiation_over_rays_and_pieces(oracle_mod, 48, 72, npieces, nray)


@pytest.mark.parametrize("heat", [0.0, 2e6])
def test_soot_too_thin_to_shine(heat):
    # an emissivity 1 - exp(-y) is an exact zero in f32 for y up to 2^-25: at and around the renderer's line for it
    # the image is the one without soot to the bit, far above the line it is not
    g = cb.FluidSim(0, {"nx": 48, "ny": 72, "dt": 1e-3}, width=0.8).init()
    g.writeParams()
    P = g.params
    T = np.full(48 * 72, 1200.0, np.float32)
    SQ = g.readBuffer("SQ").reshape(-1, 2).copy()
    SQ[:, 1] = heat
    g.writeBuffer("T", T); g.writeBuffer("SQ", SQ)
    Y = g.readBuffer("Y").reshape(-1, 4).copy()
    rho = P["rhoAmb"] * P["Tamb"] / 1200.0
    images = []
    for line in (0.0, 1e-20, 0.5, 0.99, 1.01, 1.6, 1e6):
        # y = 6.3 fv / l * depth at the shortest wavelength, 412.5 nm; fv = rho Y / sootDensity
        Y[:, 3] = line * 2.0 ** -25 * 412.5e-9 / (6.3 * P["depth"]) * P["sootDensity"] / rho
        g.writeBuffer("Y", Y)
        images.append(_image(g, 64, 96, "photo"))
    g.close()
    assert all(np.array_equal(a.view(np.uint32), images[0].view(np.uint32)) for a in images[1:-1])
    assert not np.array_equal(images[-1], images[0])
