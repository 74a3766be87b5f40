"""The step loop (a lane per path, a warp's paths in step, single-cell leaves
crossed by a loop of their own) and the pair kernel (a path's sun
transmissivity on a second warp) against the plain kernel, where the walk and
the pair's guess of the random stream can go wrong: grids of a cell or two, leaves larger than a cell, cells
that straddle gas layers (null collisions), negative coordinates and tiles,
horizontal rays, every axis consecutive in the majorant grid, and majorants
whose sign cannot mark a leaf.

One realisation per pixel, so a pixel holds one weight: both kernels take the
same draws and the same steps, and only the last FP64 operations of a weight
may be rounded differently (1e-12)."""
import numpy as np
import pytest

from htrdr_kmin_b200 import scene as S

pytestmark = pytest.mark.gpu


def _scene(nx, ny, nz, lw=False, repeat=True, lower=(-250.0, 130.0, 730.0), azimuth=30.0, elevation=60.0,
           tau=1.0, seed=5):
    z = S.layers_uniform()
    lo, hi = (8000.0, 12000.0) if lw else (500.0, 600.0)
    edges = np.linspace(lo, hi, 3)
    nq = np.full(2, 2, dtype=np.uint32)
    gas = S.gas_lw if lw else S.gas_sw
    ka, ks, w = gas(z, edges[:-1], edges[1:], nq, seed, (1e-6, 1e-3))
    full = lambda v: np.full(2, v, np.float32)  # noqa: E731
    return S.Scene(layer_z=z, layer_T=S.temperature_profile(z), band_lo=edges[:-1].copy(), band_hi=edges[1:].copy(),
                   nquads=nq, quad_w=w, gas_ka=ka, gas_ks=ks, cloud_lwc=S.lwc_power_law((nz, ny, nx), seed),
                   cloud_lower=lower, cloud_cell=(90.0, 70.0, 1000.0 / nz), cloud_sigma_ext=full(150.0),
                   cloud_ssa=full(0.999), cloud_g=full(0.85), repeat_clouds=repeat, optical_thickness=tau,
                   sun_azimuth=azimuth, sun_elevation=elevation)


def _request(lw, mode=None, **kw):
    return S.Request(**{**dict(mode=mode if mode is not None else (S.MODE_XWAVE_LW if lw else S.MODE_XWAVE_SW),
                               width=37, height=21, spp=1,
                               wlen_range=(8000.0, 12000.0) if lw else (500.0, 600.0),
                               ref_temperature=290.0 if lw else 5778.0, cam_pos=(800.0, -2500.0, 900.0),
                               cam_tgt=(800.0, 900.0, 1300.0), fov_deg=60.0, seed=11), **kw})


CASES = {
    "one_cell": (dict(nx=1, ny=1, nz=1), {}),
    "two_cells": (dict(nx=2, ny=1, nz=3), {}),
    "not_repeated": (dict(nx=19, ny=23, nz=9, repeat=False), {}),
    "straddles_layers": (dict(nx=33, ny=17, nz=5), {}),
    "large_leaves": (dict(nx=32, ny=32, nz=16, tau=60.0), {}),
    "no_merge": (dict(nx=31, ny=9, nz=7, tau=0.0), {}),
    "x_consecutive": (dict(nx=40, ny=9, nz=4, azimuth=0.0, elevation=5.0), {}),
    "y_consecutive": (dict(nx=9, ny=40, nz=4, azimuth=90.0, elevation=5.0), {}),
    "horizontal": (dict(nx=21, ny=22, nz=12), dict(camera_type=S.CAMERA_ORTHOGRAPHIC, cam_pos=(800.0, -2500.0, 1300.0),
                                                   ortho_height=800.0)),
    "lw": (dict(nx=21, ny=22, nz=12, lw=True), {}),
    "lw_large_leaves": (dict(nx=32, ny=32, nz=16, lw=True, tau=60.0), {}),
    "flux": (dict(nx=25, ny=18, nz=6), dict(mode=S.MODE_FLUX_SW, rect_pos=(500.0, 500.0, 0.0),
                                            rect_tgt=(500.0, 500.0, 1.0), rect_size=(900.0, 700.0))),
}


# 777 realisations: the pair kernel alone; 25 300: the step loop, the last paths
# handed to the pair kernel
@pytest.mark.parametrize("size", [(37, 21), (220, 115)])
@pytest.mark.parametrize("name", list(CASES))
def test_step_kernels_equal_plain(gpu_lib, name, size):
    skw, rkw = CASES[name]
    lw = skw.get("lw", False)
    gs = gpu_lib.GpuScene(_scene(**skw))
    req = _request(lw, **{**rkw, "width": size[0], "height": size[1]})
    w = gs.realisation_weights(req, 0, req.width * req.height).ravel()
    buf, st = gs.draw_map(req)
    got = (buf["sum"] if req.mode == S.MODE_FLUX_SW else buf["L"]).ravel()
    assert st["failures"] == 0 and np.count_nonzero(w) > w.size // 8
    np.testing.assert_allclose(got, w, rtol=1e-12, atol=0)


# more threads than a shortwave block has registers for, and a single warp
@pytest.mark.parametrize("block", [32, 288, 512])
@pytest.mark.parametrize("name", ["straddles_layers", "lw"])
def test_block_sizes(gpu_lib, name, block):
    skw, rkw = CASES[name]
    gs = gpu_lib.GpuScene(_scene(**skw))
    req = _request(skw.get("lw", False), **{**rkw, "width": 220, "height": 115})
    want = gs.draw_map(req)[0]["L"].ravel()
    tuning = gpu_lib.mode_tuning(req.mode)
    tuning.block_size = block
    got = gpu_lib.draw_maps_batched([(gs, req)], tuning)[0][0]["L"].ravel()
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("name", ["straddles_layers", "large_leaves", "not_repeated"])
def test_radiance_kernels_agree(gpu_lib, name):
    """A ray's radiance does not depend on how many rays the call has: the pair
    kernel (few rays) and the step loop (many)."""
    gs = gpu_lib.GpuScene(_scene(**CASES[name][0]))
    rng = np.random.default_rng(2)
    n = 45000
    pos = rng.uniform((0, 0, 1), (1800, 1300, 2500), (n, 3))
    d = rng.standard_normal((n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    band = rng.integers(0, 2, n).astype(np.uint32)
    quad = rng.integers(0, 2, n).astype(np.uint32)
    wlen = 525.0 + 50.0 * band
    many = gs.radiance_sw(pos, d, wlen, band, quad, seed=4)
    for k in (1, 33, 6000):
        few = gs.radiance_sw(pos[:k], d[:k], wlen[:k], band[:k], quad[:k], seed=4)
        np.testing.assert_allclose(few, many[:k], rtol=1e-12, atol=0)


def test_negative_majorants_take_the_general_voxel(gpu_lib):
    """A majorant below zero (a medium no user means, but one that is
    accepted) leaves no sign to mark leaves with: every voxel by the general
    step, with the plain kernel's sums."""
    sc = _scene(nx=12, ny=10, nz=6)
    sc.cloud_lwc = sc.cloud_lwc.copy()
    sc.cloud_lwc[:, :5, :] = 0.0
    sc.cloud_lwc[2, 2, 3] = -1e-6
    gs = gpu_lib.GpuScene(sc)
    assert min(gs.tree(0, 0, gpu_lib.KEXT)["kmax"].min(), gs.tree(0, 0, gpu_lib.KS)["kmin"].min()) < 0
    req = _request(False)
    w = gs.realisation_weights(req, 0, req.width * req.height).ravel()
    buf, _ = gs.draw_map(req)
    ok = np.isfinite(w)
    np.testing.assert_allclose(buf["L"].ravel()[ok], w[ok], rtol=1e-12, atol=0)
