"""Performance cases of the atmosphere path tracer: the calls a user of the
library makes, over the range of sizes it is used at, through the package's
public entry points.

A case is a dict of plain values; `kind` names the entry point:

* ``map``: ``GpuScene.draw_map`` (htrdr_draw_map), one image or flux map into
  a host buffer, on the engine the library picks by itself;
* ``batch``: ``draw_maps_batched``, uneven image requests on three scenes;
* ``serve``: ``Server.submit`` / ``wait``, the same mix through the request
  loop;
* ``radiance``: ``GpuScene.radiance_sw`` / ``radiance_lw``, one ray per
  radiance estimate;
* ``create``: ``GpuScene(...)`` (htsky_create), the upload of a medium and the
  build of its majorant octrees.

Scenes follow the recipes of the package's own workloads (scene.config_c1,
config_c2, config_c3, batched_scenes): 50 gas layers up to 50 km, a 1 km
thick cloud based at 1 km, lognormal or k^-5/3 liquid water, droplet albedo
0.999 and asymmetry 0.85.  The medium, the random streams and the rays all
come from the seed.

Outputs are the maps' estimators, radiances and octree nodes.  The per-pixel
sums of the time spent on each realisation (``t_sum``, ``t_sum2``) are clock
readings and are left out.  ``exact`` has no value to give: an estimate is a
Monte Carlo sum whose terms are picked by the single-precision walk itself,
and a majorant octree's shape by single-precision comparisons.
"""
from __future__ import annotations

import math

import numpy as np

from htrdr_kmin_b200 import api
from htrdr_kmin_b200 import scene as S

MODES = {"sw_image": S.MODE_XWAVE_SW, "lw_image": S.MODE_XWAVE_LW, "cie_image": S.MODE_IMAGE_CIE,
         "sw_flux": S.MODE_FLUX_SW, "lw_flux": S.MODE_FLUX_LW}
RANGES = {"sw": (500.0, 600.0), "cie": (380.0, 780.0), "lw": (3000.0, 100000.0)}
LAYERS = 50


def listed():
    return [
        # a look at a scene while its camera is being placed: the smallest call
        dict(name="sw_preview", kind="map", mode="sw_image", nx=32, ny=32, nz=16, field="lognormal",
             cell=100.0, repeat=False, nbands=1, nquads=1, width=16, height=16, spp=4, mesh=False),
        # the shortwave image of the small configuration (64 x 64 px, 32 realisations)
        dict(name="sw_image", kind="map", mode="sw_image", nx=32, ny=32, nz=16, field="lognormal",
             cell=100.0, repeat=False, nbands=1, nquads=1, width=64, height=64, spp=32, mesh=False),
        # a radiance image in the thermal infrared, odd image and cloud sizes
        dict(name="lw_image", kind="map", mode="lw_image", nx=97, ny=83, nz=37, field="power",
             cell=50.0, repeat=True, nbands=16, nquads=8, width=251, height=187, spp=48, mesh=False),
        # the longwave flux map of the second configuration: the largest number of realisations
        dict(name="lw_flux", kind="map", mode="lw_flux", nx=64, ny=64, nz=32, field="lognormal",
             cell=100.0, repeat=True, nbands=16, nquads=8, width=128, height=128, spp=256, mesh=False),
        # solar flux at the ground under an infinitely repeated cloud field
        dict(name="sw_flux", kind="map", mode="sw_flux", nx=64, ny=48, nz=32, field="power",
             cell=100.0, repeat=True, nbands=4, nquads=4, width=61, height=45, spp=32, mesh=False),
        # a colour image: three channels, many bands
        dict(name="cie_image", kind="map", mode="cie_image", nx=128, ny=128, nz=32, field="power",
             cell=50.0, repeat=False, nbands=15, nquads=8, width=128, height=96, spp=8, mesh=False),
        # a shortwave image over a terrain mesh of two materials
        dict(name="mesh_image", kind="map", mode="sw_image", nx=48, ny=40, nz=24, field="lognormal",
             cell=80.0, repeat=True, nbands=2, nquads=2, width=72, height=54, spp=16, mesh=True),
        # uneven requests on three scenes in one call (the headline workload at half scale)
        dict(name="batch_mix", kind="batch", scale=0.5, requests=32, side_lo=16, side_hi=64, spp_lo=16,
             spp_hi=64),
        # the same kind of requests arriving together at the request loop
        dict(name="serve_mix", kind="serve", scale=0.25, requests=24, side_lo=8, side_hi=64, spp_lo=8,
             spp_hi=64),
        # radiance estimates for a caller's own rays
        dict(name="radiance_sw", kind="radiance", lw=False, nx=64, ny=64, nz=32, field="power", cell=50.0,
             repeat=True, nbands=4, nquads=4, n=20000),
        dict(name="radiance_lw", kind="radiance", lw=True, nx=64, ny=64, nz=32, field="power", cell=50.0,
             repeat=True, nbands=16, nquads=8, n=300001),
        # opening a scene: upload and octrees of 32 quadrature points, all three properties
        dict(name="scene_create", kind="create", nx=112, ny=90, nz=40, field="power", cell=50.0,
             repeat=False, nbands=8, nquads=4),
    ]


def _logu(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["map", "batch", "serve", "radiance", "create"], [6, 1, 1, 2, 1])[0]
    if kind in ("batch", "serve"):
        return dict(kind=kind, scale=round(rng.uniform(0.15, 0.4), 3), requests=rng.randint(4, 24),
                    side_lo=8, side_hi=rng.randint(24, 64), spp_lo=8, spp_hi=rng.randint(24, 64))
    c = dict(kind=kind, nx=_logu(rng, 12, 128), ny=_logu(rng, 12, 128), nz=_logu(rng, 8, 48),
             field=rng.choice(["lognormal", "power"]), cell=rng.choice([50.0, 75.0, 100.0]),
             repeat=rng.random() < 0.5)
    if kind == "create":
        c.update(nbands=rng.randint(1, 6), nquads=rng.randint(1, 6))
        return c
    if kind == "radiance":
        lw = rng.random() < 0.5
        c.update(lw=lw, nbands=rng.randint(1, 12), nquads=rng.randint(1, 8),
                 n=_logu(rng, 100, 300000 if lw else 20000))
        return c
    mode = rng.choice(list(MODES))
    lw = mode in ("lw_image", "lw_flux")
    # realisations log-uniform, then split between pixels and samples
    real = _logu(rng, 1000, 4000000 if lw else 130000)
    spp = _logu(rng, 4, 64)
    ratio = rng.uniform(0.6, 1.6)
    per_px = spp * (3 if mode == "cie_image" else 1)
    width = max(3, int(round(math.sqrt(real / per_px * ratio))))
    height = max(3, int(round(real / per_px / width)))
    c.update(mode=mode, nbands=rng.randint(1, 16 if lw else 6), nquads=rng.randint(1, 8), width=width,
             height=height, spp=spp, mesh=mode in ("sw_image", "lw_image") and rng.random() < 0.25)
    return c


# ---- what the caller holds before the call ---------------------------------
def _scene(c, domain, seed):
    """Medium of a case: gas column, cloud, optics, ground, sun."""
    z = S.layers_uniform(n=LAYERS)
    nb = c["nbands"]
    lo, hi = RANGES[domain]
    edges = np.geomspace(lo, hi, nb + 1) if domain == "lw" else np.linspace(lo, hi, nb + 1)
    edges[0], edges[-1] = lo, hi
    nq = np.full(nb, c["nquads"], dtype=np.uint32)
    gas = S.gas_lw if domain == "lw" else S.gas_sw
    ka, ks, w = gas(z, edges[:-1], edges[1:], nq, seed * 8 + 1)
    lwc = (S.lwc_lognormal if c["field"] == "lognormal" else S.lwc_power_law)(
        (c["nz"], c["ny"], c["nx"]), seed * 8 + 2)
    full = lambda v: np.full(nb, v, dtype=np.float32)  # noqa: E731
    sc = S.Scene(layer_z=z, layer_T=S.temperature_profile(z), band_lo=edges[:-1].copy(),
                 band_hi=edges[1:].copy(), nquads=nq, quad_w=w, gas_ka=ka, gas_ks=ks, cloud_lwc=lwc,
                 cloud_lower=(0.0, 0.0, 1000.0), cloud_cell=(c["cell"], c["cell"], 1000.0 / c["nz"]),
                 cloud_sigma_ext=full(S.SIGMA_EXT_CLOUD), cloud_ssa=full(0.999), cloud_g=full(0.85),
                 repeat_clouds=c["repeat"], ground_reflectivity=0.05 if domain == "lw" else 0.2,
                 sun_azimuth=30.0, sun_elevation=60.0)
    if c.get("mesh"):
        sc = S.with_terrain(sc, size=c["nx"] * c["cell"], n=24, amp=150.0, seed=seed * 8 + 3, repeat=True)
    return sc


def _request(c, seed):
    """Sensor of a map case, over the cloud field's extent."""
    mode = c["mode"]
    ex, ey = c["nx"] * c["cell"], c["ny"] * c["cell"]
    lw = mode in ("lw_image", "lw_flux")
    rq = dict(mode=MODES[mode], width=c["width"], height=c["height"], spp=c["spp"],
              wlen_range=RANGES["lw" if lw else ("cie" if mode == "cie_image" else "sw")],
              ref_temperature=290.0 if lw else 5778.0, seed=seed & 0x7FFFFFFF)
    if mode in ("sw_flux", "lw_flux"):
        rq.update(rect_pos=(0.5 * ex, 0.5 * ey, 0.0), rect_tgt=(0.5 * ex, 0.5 * ey, 1.0),
                  rect_up=(0.0, 1.0, 0.0), rect_size=(ex, ey))
    elif mode == "lw_image":  # from above the ground, towards the sky
        rq.update(cam_pos=(0.5 * ex, 0.5 * ey, 200.0), cam_tgt=(0.5 * ex + 100.0, 0.5 * ey + 100.0, 3000.0),
                  fov_deg=60.0)
    else:  # from the side, across the cloud field
        rq.update(cam_pos=(0.5 * ex, -0.9 * ey, 900.0), cam_tgt=(0.5 * ex, 0.5 * ey, 1500.0), fov_deg=60.0)
    return S.Request(**rq)


def _mix(c, seed):
    """Three scenes and the uneven requests on them (half shortwave images,
    half longwave images)."""
    scenes = []
    for i, sc in enumerate(S.batched_scenes(c["scale"])):
        sc.cloud_lwc = S.lwc_power_law(sc.cloud_lwc.shape, seed * 8 + i)
        scenes.append(api.GpuScene(sc))
    # sizes belong to the case, streams to the seed
    reqs = S.batched_requests(c["requests"], seed=4, side_range=(c["side_lo"], c["side_hi"]),
                              spp_range=(c["spp_lo"], c["spp_hi"]))
    items = []
    for k, (i, rq) in enumerate(reqs):
        rq.seed = (seed * 1000 + k) & 0x7FFFFFFF
        items.append((scenes[i], rq))
    return items


def _domain(c):
    if c["kind"] == "radiance":
        return "lw" if c["lw"] else "sw"
    return {"lw_image": "lw", "lw_flux": "lw", "cie_image": "cie"}.get(c.get("mode"), "sw")


def prepare(case, seed):
    kind = case["kind"]
    if kind == "create":
        # nodes of an octree without a merged leaf: room for any tree of the grid
        dims, nodes = [case["nx"], case["ny"], case["nz"]], 1
        while max(dims) > 1:
            dims = [(d + 1) // 2 for d in dims]
            nodes += 8 * dims[0] * dims[1] * dims[2]
        return dict(kind=kind, scene=_scene(case, "sw", seed), nodes=nodes)
    if kind in ("batch", "serve"):
        st = dict(kind=kind, items=_mix(case, seed))
        if kind == "serve":
            st["server"] = api.Server(tuning=api.mode_tuning(S.MODE_XWAVE_SW))
        return st
    sc = _scene(case, _domain(case), seed)
    if kind == "map":
        rq = _request(case, seed)
        return dict(kind=kind, scene=api.GpuScene(sc, props_mask=api.props_for_mode(rq.mode)), req=rq)
    rng = np.random.default_rng(seed)
    n = case["n"]
    ex, ey = case["nx"] * case["cell"], case["ny"] * case["cell"]
    pos = np.stack([rng.uniform(0, ex, n), rng.uniform(0, ey, n), rng.uniform(1.0, 3000.0, n)], axis=1)
    d = rng.standard_normal((n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    band = rng.integers(0, case["nbands"], n).astype(np.uint32)
    quad = rng.integers(0, case["nquads"], n).astype(np.uint32)
    wlen = 0.5 * (sc.band_lo[band] + sc.band_hi[band])
    mode = S.MODE_XWAVE_LW if case["lw"] else S.MODE_XWAVE_SW
    return dict(kind=kind, scene=api.GpuScene(sc, props_mask=api.props_for_mode(mode)),
                rays=(pos, d, wlen, band, quad), lw=case["lw"], seed=seed & 0x7FFFFFFF)


def _values(buf):
    """A map's estimators: every field but the clock readings."""
    return {f: np.ascontiguousarray(buf[f]) for f in buf.dtype.names if f not in ("t_sum", "t_sum2")}


def _together(bufs):
    """The estimators of several image maps, one after another."""
    maps = [_values(b) for b in bufs]
    return {f: np.concatenate([m[f].reshape(-1) for m in maps]) for f in maps[0]}


def run(state):
    kind = state["kind"]
    if kind == "map":
        buf, _ = state["scene"].draw_map(state["req"])
        return _values(buf)
    if kind == "batch":
        bufs, _ = api.draw_maps_batched(state["items"])
        return _together(bufs)
    if kind == "serve":
        tickets = [state["server"].submit(gs, rq) for gs, rq in state["items"]]
        return _together([state["server"].wait(t) for t in tickets])
    if kind == "radiance":
        call = state["scene"].radiance_lw if state["lw"] else state["scene"].radiance_sw
        return call(*state["rays"], seed=state["seed"])
    scene = api.GpuScene(state["scene"])
    out = {"depth": scene.depth()}
    for prop in (api.KA, api.KS, api.KEXT):
        nodes = np.zeros(state["nodes"], dtype=api.NODE_DTYPE)
        t = scene.tree(0, 0, prop)
        nodes[:len(t)] = t
        out["prop%d" % prop] = {f: np.ascontiguousarray(nodes[f]) for f in ("kmin", "kmax", "child")}
    scene.close()
    return out


def exact(case, seed):
    return None


# ---- what a pass cannot do without -----------------------------------------
# Voxels a realisation crosses on average (the library's own counters on the
# package's workloads) and floating-point operations of one crossing: three
# plane distances, the optical depth, the next cell.
VOXELS = {"sw": 1500.0, "lw": 15.0}
FLOPS_PER_VOXEL = 40.0


def work(case):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        reqs = S.batched_requests(case["requests"], seed=4, side_range=(case["side_lo"], case["side_hi"]),
                                  spp_range=(case["spp_lo"], case["spp_hi"]))
        cells = sum(a * b * d for a, b, d in
                    (tuple(max(2, int(round(v * case["scale"]))) for v in t)
                     for t in ((128, 128, 128), (256, 256, 64), (512, 512, 128))))
        vox = sum(r.realisations * VOXELS["lw" if r.mode == S.MODE_XWAVE_LW else "sw"] for _, r in reqs)
        return {"bytes": 4.0 * cells + 3 * 32 * LAYERS * 8.0 + sum(r.width * r.height * 64.0 for _, r in reqs),
                "flops": vox * FLOPS_PER_VOXEL}
    cells = case["nx"] * case["ny"] * case["nz"]
    nq = case["nbands"] * case["nquads"]
    medium = 4.0 * cells + nq * LAYERS * 8.0
    if kind == "create":  # the medium in, kmin and kmax of every cell of every property's octree out
        return {"bytes": medium + nq * 3 * cells * 8.0, "flops": nq * 3 * cells * 4.0}
    lw = _domain(case) == "lw"
    if kind == "radiance":
        real, io = case["n"], case["n"] * (7 * 8 + 8 + 8.0)
    else:
        real = case["width"] * case["height"] * case["spp"] * (3 if case["mode"] == "cie_image" else 1)
        io = case["width"] * case["height"] * (80.0 if case["mode"] == "cie_image" else 64.0)
    return {"bytes": medium + io, "flops": real * VOXELS["lw" if lw else "sw"] * FLOPS_PER_VOXEL}
