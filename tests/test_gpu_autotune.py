"""What the autotuner returns can be used wherever a tuning is taken."""
import ctypes as C

import numpy as np
import pytest

from htrdr_kmin_b200 import scene as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["sw", "lw"])
def test_autotuned_tuning_is_taken_everywhere(gpu_lib, mode):
    import torch
    api = gpu_lib
    sc, rq = S.config_c1(scale=16 / 64, spp=4) if mode == "sw" else S.config_c2(scale=16 / 128, spp=4,
                                                                               cloud_def=(16, 16, 8))
    gs = api.GpuScene(sc)
    want = gs.draw_map(rq)[0]
    key = "L" if mode == "sw" else "sum"
    dev = torch.zeros(want.nbytes, dtype=torch.uint8, device="cuda:0")
    arr = (api.BatchItem * 1)()
    arr[0].scene, arr[0].req, arr[0].layout = gs.handle.value, api.to_request(rq), api.layout_for(rq)
    arr[0].buffer = dev.data_ptr()
    tuning, ms = api.autotune(arr)
    assert ms > 0
    got = api.draw_maps_batched([(gs, rq)], tuning)[0][0]
    np.testing.assert_allclose(got[key], want[key], rtol=1e-9, atol=0)
    h = C.c_void_p()
    L = api.lib()
    assert L.htrdr_gpu_batch_create(arr, 1, C.byref(tuning), C.byref(h)) == 0, L.htrdr_gpu_last_error()
    dev.zero_()
    torch.cuda.synchronize()
    assert L.htrdr_gpu_batch_run(h, C.byref(api.Stats())) == 0
    got = np.frombuffer(dev.cpu().numpy().tobytes(), dtype=want.dtype).reshape(want.shape)
    L.htrdr_gpu_batch_release(h)
    np.testing.assert_allclose(got[key], want[key], rtol=1e-9, atol=0)
    srv = api.Server(tuning=tuning)
    got = srv.wait(srv.submit(gs, rq), 120.0)
    srv.close()
    np.testing.assert_allclose(got[key], want[key], rtol=1e-9, atol=0)
    gs.set_engine(tuning.engine, tuning)
    np.testing.assert_allclose(gs.draw_map(rq)[0][key], want[key], rtol=1e-9, atol=0)
