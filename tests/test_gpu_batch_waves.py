"""The automatic waves of a batch: split so that film copies overlap the render
where several jobs have host films, whole where nothing would be gained."""
import ctypes as C

import numpy as np
import pytest

from pyre_gb300 import native as N
from pyre_gb300 import presets as P

pytestmark = pytest.mark.gpu

W, H, SPP = 768, 512, 48  # 18.9 M samples a job: two of them are more than 32 Mi


@pytest.mark.parametrize("jobs,mem,waves", [(1, "host", 1), (2, "host", 2), (2, "device", 1), (3, "device", 1)])
def test_waves_of_a_batch(gpu_ctx, jobs, mem, waves):
    import torch
    ds = gpu_ctx.upload_batch([P.cornell_box()])
    dev = [torch.zeros((H, W, 3), device="cuda") for _ in range(jobs)]
    host = [np.zeros((H, W, 3), np.float32) for _ in range(jobs)]
    arr = (N.BatchJob * jobs)()
    for b, d, h in zip(arr, dev, host):
        b.part, b.camera, b.width, b.height, b.spp_end = 0, P.cornell_box_camera(W, H).to_desc(), W, H, SPP * 2 // jobs
        b.max_depth, b.min_rr_depth = 1, 1
        b.film = (N.Film(N.dptr(d), None, None, None, N.PYRE_MEM_DEVICE) if mem == "device"
                  else N.Film(N.fptr(h), None, None, None, N.PYRE_MEM_HOST))
    p = N.RenderParams()
    gpu_ctx.check(gpu_ctx.lib.pyre_render_batch(gpu_ctx.handle, ds.handle, arr, jobs, C.byref(p)))
    s = gpu_ctx.stats()
    assert s.samples == jobs * W * H * (SPP * 2 // jobs) and s.samples > 32 << 20
    assert s.waves == waves
    ds.close()
