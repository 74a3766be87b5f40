"""The batched octree build on the GPU against the host build, node for node,
where its Morton ranks can go wrong: one cell, skinny and odd grids (levels
whose coordinates have different numbers of bits), no merged leaf, all merged,
the -V cap, and properties left out.  Byte equality: both are the same
single-precision operations and the same order."""
import numpy as np
import pytest

from htrdr_kmin_b200 import scene as S

pytestmark = pytest.mark.gpu


def _scene(nx, ny, nz, tau, vmax, lower):
    z = S.layers_uniform(top=20000.0, n=23)
    edges = np.linspace(500.0, 600.0, 3)
    nq = np.array([2, 1], dtype=np.uint32)
    ka, ks, w = S.gas_sw(z, edges[:-1], edges[1:], nq, 3)
    full = lambda v: np.full(2, v, np.float32)  # noqa: E731
    return S.Scene(layer_z=z, layer_T=S.temperature_profile(z), band_lo=edges[:-1].copy(), band_hi=edges[1:].copy(),
                   nquads=nq, quad_w=w, gas_ka=ka, gas_ks=ks, cloud_lwc=S.lwc_lognormal((nz, ny, nx), 8, 0.05, 1.5),
                   cloud_lower=(0.0, 0.0, lower), cloud_cell=(60.0, 50.0, 40.0), cloud_sigma_ext=full(150.0),
                   cloud_ssa=full(0.9), cloud_g=full(0.85), optical_thickness=tau, grid_max_definition=vmax)


@pytest.mark.parametrize("shape,tau,vmax", [
    ((1, 1, 1), 1.0, (0, 0, 0)), ((2, 1, 1), 0.0, (0, 0, 0)), ((1, 1, 9), 0.5, (0, 0, 0)),
    ((1000, 1, 2), 0.5, (0, 0, 0)), ((3, 257, 5), 0.5, (0, 0, 0)), ((33, 16, 7), 0.0, (0, 0, 0)),
    ((31, 64, 15), 1e9, (0, 0, 0)), ((64, 64, 32), 1.0, (16, 0, 0)), ((65, 3, 33), 2.0, (0, 0, 8))])
@pytest.mark.parametrize("props", [0b111, 0b100])
def test_gpu_build_equals_host_build(gpu_lib, shape, tau, vmax, props):
    sc = _scene(*shape, tau, vmax, lower=830.0)
    g, h = gpu_lib.GpuScene(sc, props), gpu_lib.GpuScene(sc, props, octree_on_host=True)
    for band, quad in ((0, 0), (0, 1), (1, 0)):
        for p in range(3):
            a, b = g.tree(band, quad, p), h.tree(band, quad, p)
            assert len(a) == len(b) and (len(a) > 0) == bool(props >> p & 1)
            assert a.tobytes() == b.tobytes()
