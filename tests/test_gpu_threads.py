"""Host threads that call the library at once: what one launches must not
depend on what another does."""
import threading

import numpy as np
import pytest

from htrdr_kmin_b200 import scene as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", ["step", "sorted"])
def test_batches_and_maps_at_once(gpu_lib, engine):
    """Launches of the same kernels with tables of one request and of up to
    120: their shared memory differs, and each is granted its own."""
    api = gpu_lib
    sc, rq = S.config_c1(scale=6 / 64, spp=1)
    tuning = api.mode_tuning(rq.mode)
    if engine == "sorted":
        tuning.engine = api.ENGINE_SORTED
    scenes = [api.GpuScene(sc) for _ in range(2)]
    reqs = [S.Request(**{**rq.__dict__, "seed": 10 + i}) for i in range(120)]
    want = [scenes[0].draw_map(r)[0]["L"] for r in reqs]
    errors = []

    def draw(gs, sizes, calls):
        try:
            for k in range(calls):
                n = sizes[k % len(sizes)]
                bufs, _ = api.draw_maps_batched([(gs, r) for r in reqs[:n]], tuning)
                for b, w in zip(bufs, want):
                    np.testing.assert_allclose(b["L"], w, rtol=1e-9, atol=0)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=draw, args=(scenes[0], (1,), 300)),
               threading.Thread(target=draw, args=(scenes[1], (120, 7, 60), 300))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
