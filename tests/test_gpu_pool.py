"""The serving pool beside other work on the device, and at the ends of its
settings.  A request's map is the one drawn alone (1e-9 relative: the FP64
summation order)."""
import threading

import numpy as np
import pytest

from htrdr_kmin_b200 import scene as S

pytestmark = pytest.mark.gpu

RTOL = 1e-9
WAIT_S = 120.0


def _estimates(buf, mode):
    return buf["sum"] if mode in (S.MODE_FLUX_SW, S.MODE_FLUX_LW) else buf["L"]


def _same(a, b, mode):
    np.testing.assert_allclose(_estimates(a, mode), _estimates(b, mode), rtol=RTOL, atol=0)
    np.testing.assert_array_equal(a["t_n"], b["t_n"])


def _requests(api):
    s1, r1 = S.config_c1(scale=16 / 64, spp=16)
    s2, r2 = S.config_c2(scale=32 / 128, spp=16, cloud_def=(16, 16, 8))
    scenes = [(api.GpuScene(s1), r1), (api.GpuScene(s2, 0b100), r2)]
    out = []
    for i in range(16):
        gs, r = scenes[i % 2]
        side = (12, 40, 25, 33)[i % 4]
        out.append((gs, S.Request(**{**r.__dict__, "width": side, "height": side + 1, "spp": (4, 8, 3)[i % 3],
                                     "seed": 300 + i})))
    return out


def _pool(api, slots=0, **kw):
    t = api.mode_tuning(S.MODE_XWAVE_SW)
    t.wave_slots = slots
    return api.Server(tuning=t, **kw)


# pools of fewer paths than warps, of about one a warp, and as large as they get
@pytest.mark.parametrize("slots", [37, 1500, 0])
def test_pool_beside_other_calls(gpu_lib, slots):
    """Blocks of the pool's launches that start late, as other calls hold the
    SMs: no path is lost, none is kept twice, none has no room."""
    api = gpu_lib
    reqs = _requests(api)
    alone = [gs.draw_map(r)[0] for gs, r in reqs]
    sc, rq = S.config_c1(scale=0.5, spp=32)
    other = api.GpuScene(sc)
    want = other.draw_map(rq)[0]
    over = threading.Event()
    maps = []

    def draw():
        while not over.is_set():
            maps.append(other.draw_map(rq)[0])

    srv = _pool(api, slots)
    th = threading.Thread(target=draw)
    th.start()
    try:
        for _ in range(3):
            tickets = [srv.submit(*it) for it in reqs]
            out = [srv.wait(t, WAIT_S) for t in tickets]
            for (gs, r), a, b in zip(reqs, out, alone):
                _same(a, b, r.mode)
    finally:
        over.set()
        th.join()
    st = srv.stats()
    srv.close()
    assert st["failed"] == 0 and maps
    for m in maps:
        _same(m, want, rq.mode)


@pytest.mark.parametrize("target_ms", [1e-5, 1e9])
def test_pool_advances_whatever_the_round_target(gpu_lib, target_ms):
    api = gpu_lib
    reqs = _requests(api)[:6]
    srv = _pool(api, round_target_ms=target_ms)
    tickets = [srv.submit(*it) for it in reqs]
    out = [srv.wait(t, WAIT_S) for t in tickets]
    srv.close()
    for (gs, r), a in zip(reqs, out):
        _same(a, gs.draw_map(r)[0], r.mode)
