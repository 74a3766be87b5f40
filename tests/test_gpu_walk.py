"""The walk through single-cell leaves and the kernels' hand-over where the
scene or the run differs from the usual one, against the plain kernel."""
import numpy as np
import pytest

from htrdr_kmin_b200 import scene as S

pytestmark = pytest.mark.gpu


def _scene(nx=33, ny=29, nz=12, nbands=2, nquads=2, lw=False, mesh=False, cloud=None, tau=1.0, seed=9):
    z = S.layers_uniform()
    lo, hi = (8000.0, 12000.0) if lw else (500.0, 600.0)
    edges = np.linspace(lo, hi, nbands + 1)
    nq = np.full(nbands, nquads, dtype=np.uint32)
    ka, ks, w = (S.gas_lw if lw else S.gas_sw)(z, edges[:-1], edges[1:], nq, seed, (1e-6, 1e-3))
    lwc = S.lwc_power_law((nz, ny, nx), seed)
    if cloud is not None:  # liquid water in a corner of the grid only
        lwc[:, cloud:, :] = 0.0
        lwc[:, :, cloud:] = 0.0
    full = lambda v: np.full(nbands, v, np.float32)  # noqa: E731
    sc = S.Scene(layer_z=z, layer_T=S.temperature_profile(z), band_lo=edges[:-1].copy(), band_hi=edges[1:].copy(),
                 nquads=nq, quad_w=w, gas_ka=ka, gas_ks=ks, cloud_lwc=lwc, cloud_lower=(0.0, 0.0, 1000.0),
                 cloud_cell=(80.0, 80.0, 1000.0 / nz), cloud_sigma_ext=full(150.0), cloud_ssa=full(0.99),
                 cloud_g=full(0.85), repeat_clouds=True, optical_thickness=tau, sun_azimuth=30.0,
                 sun_elevation=40.0)
    return S.with_terrain(sc, size=nx * 80.0, n=12, amp=150.0, seed=3, repeat=True) if mesh else sc


def _request(mode=S.MODE_XWAVE_SW, width=37, height=21, spp=1, seed=11):
    lw = mode == S.MODE_XWAVE_LW
    return S.Request(mode=mode, width=width, height=height, spp=spp,
                     wlen_range=(8000.0, 12000.0) if lw else (500.0, 600.0),
                     ref_temperature=290.0 if lw else 5778.0, cam_pos=(800.0, -2500.0, 900.0),
                     cam_tgt=(800.0, 900.0, 1300.0), fov_deg=60.0, seed=seed)


def _plain(api, gs, req):
    gs.set_engine(api.ENGINE_PLAIN)
    buf, st = gs.draw_map(req)
    gs.set_engine(api.ENGINE_PERSISTENT)
    return buf, st


@pytest.mark.parametrize("size", [(37, 21), (220, 115)])
def test_leaves_without_extinction(gpu_lib, size):
    """A gas that does not absorb: the absorption trees' leaves outside the
    cloud are large and hold 0, whose sign still marks them as large."""
    sc = _scene(cloud=15)
    sc.gas_ka = np.zeros_like(sc.gas_ka)
    gs = gpu_lib.GpuScene(sc)
    req = _request(width=size[0], height=size[1])
    want, sw = _plain(gpu_lib, gs, req)
    got, st = gs.draw_map(req)
    np.testing.assert_allclose(got["L"], want["L"], rtol=1e-12, atol=0)
    for k in ("segments", "collisions", "nodes", "grid_bytes", "realisations"):
        assert st[k] == sw[k], k


def test_grid_bytes_of_single_cells(gpu_lib):
    """No leaf larger than a cell (no two cells with the same liquid water, no
    merging): 8 bytes for each voxel of the cloud."""
    sc = _scene(nx=32, ny=28, nz=12, tau=0.0)
    sc.cloud_lwc = np.random.default_rng(1).uniform(1e-4, 1e-3, sc.cloud_lwc.shape).astype(np.float32)
    gs = gpu_lib.GpuScene(sc)
    req = _request(width=220, height=115)
    want, sw = _plain(gpu_lib, gs, req)
    got, st = gs.draw_map(req)
    assert 0 < st["grid_bytes"] <= 8 * st["segments"] and st["grid_bytes"] % 8 == 0
    assert st["grid_bytes"] == sw["grid_bytes"]


def _exact(api, gs, req, buf):
    """One realisation a pixel: the map holds the plain kernel's weights."""
    w = gs.realisation_weights(req, 0, req.width * req.height).ravel()
    assert np.count_nonzero(w) > w.size // 8
    np.testing.assert_allclose(buf["L"].ravel(), w, rtol=1e-12, atol=0)


# the pair kernel alone; the step loop, its last paths in the pair kernel
@pytest.mark.parametrize("size", [(37, 21), (220, 115)])
def test_mesh_and_its_last_paths(gpu_lib, size):
    gs = gpu_lib.GpuScene(_scene(mesh=True))
    req = _request(width=size[0], height=size[1])
    buf, st = gs.draw_map(req)
    assert st["failures"] == 0
    _exact(gpu_lib, gs, req, buf)


@pytest.mark.parametrize("mesh", [False, True])
def test_mixed_kinds_and_their_last_paths(gpu_lib, mesh):
    """Shortwave and longwave requests in one queue, more than the pair
    kernel's lanes, in an order that the queue does not keep."""
    sw, lw = gpu_lib.GpuScene(_scene(mesh=mesh)), gpu_lib.GpuScene(_scene(lw=True), 0b100)
    items = [(lw, _request(S.MODE_XWAVE_LW, 90, 70, seed=1)), (sw, _request(S.MODE_XWAVE_SW, 150, 90, seed=2)),
             (lw, _request(S.MODE_XWAVE_LW, 11, 9, seed=3)), (sw, _request(S.MODE_XWAVE_SW, 101, 99, seed=4))]
    assert sum(r.width * r.height for _, r in items) > 18944
    bufs, st = gpu_lib.draw_maps_batched(items)
    assert st["failures"] == 0
    for (gs, req), buf in zip(items, bufs):
        _exact(gpu_lib, gs, req, buf)


@pytest.mark.parametrize("grid", ["nodes", "none"])
def test_scenes_without_a_majorant_grid(gpu_lib, grid):
    """A scene whose majorant grid (9 bytes a cell and tree) is more than half
    of the free memory gets the node grid (4 bytes), or none: its maps are
    those of the same scene created with room for all."""
    import torch
    kw = dict(nx=128, ny=128, nz=32, nbands=8, nquads=4, cloud=20)  # 96 trees: 453 and 201 MB
    sc = _scene(**kw)
    roomy = gpu_lib.GpuScene(sc)
    free = torch.cuda.mem_get_info()[0]
    room = (650 if grid == "nodes" else 330) << 20
    hog = torch.empty(free - room, dtype=torch.uint8, device="cuda:0")
    try:
        gs = gpu_lib.GpuScene(sc)
        cells = 128 * 128 * 32 * 96
        # without any grid, no ranks of the trees' grids (4 bytes a tree) either
        assert roomy.device_bytes - gs.device_bytes == (cells * 5 if grid == "nodes" else cells * 9 + 96 * 4)
        for size in ((37, 21), (220, 115)):
            req = _request(width=size[0], height=size[1])
            buf, st = gs.draw_map(req)
            assert st["failures"] == 0 and (st["grid_bytes"] > 0) == (grid == "nodes")
            _exact(gpu_lib, roomy, req, buf)
            _exact(gpu_lib, gs, req, buf)
        gs.close()
    finally:
        del hog
        torch.cuda.empty_cache()


@pytest.mark.parametrize("grid", ["nodes", "none"])
def test_longwave_without_a_majorant_grid(gpu_lib, grid):
    """As above, for longwave paths: two voxels of the cloud a turn."""
    import torch
    sc = _scene(nx=128, ny=128, nz=32, nbands=8, nquads=4, cloud=100, tau=30.0, lw=True)  # 96 trees
    room = (700 if grid == "nodes" else 380) << 20
    hog = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda:0")
    try:
        gs = gpu_lib.GpuScene(sc)
        for size in ((37, 21), (220, 115)):
            req = _request(S.MODE_XWAVE_LW, *size)
            want, sw = _plain(gpu_lib, gs, req)
            buf, st = gs.draw_map(req)
            assert st["failures"] == 0 and (st["grid_bytes"] > 0) == (grid == "nodes")
            for k in ("segments", "nodes", "collisions", "grid_bytes"):
                assert st[k] == sw[k], k
            np.testing.assert_allclose(buf["L"], want["L"], rtol=1e-12, atol=0)
        gs.close()
    finally:
        del hog
        torch.cuda.empty_cache()
