"""block_size is a launch knob: films keep their bits, and a small block costs
little. The traversals keep their own blocks; with blocks of 32 threads and the
shared memory of 128 each, they ran with half the warps and a render took 1.5 to
1.6 times as long, where the other stages alone cost a few per cent."""
import numpy as np
import pytest

from pyre_gb300 import native as N
from pyre_gb300 import presets as P
from pyre_gb300.scene import PathIntegrator

pytestmark = pytest.mark.gpu


def _render(ctx, ds, cam, w, h, spp, width, block):
    import torch
    rad = torch.zeros((h, w, 3), device="cuda")
    film = N.Film(N.dptr(rad), None, None, None, N.PYRE_MEM_DEVICE)
    p = ctx.params(w, h, 0, spp, PathIntegrator(8, 3), block_size=block, bvh_width=width)
    ms = []
    for _ in range(5):
        ctx.render_into(ds, cam, p, film)
        ms.append(ctx.stats().ms_total)
    return rad.cpu().numpy(), min(ms[1:])


@pytest.mark.parametrize("width", [2, 4])
def test_block_sizes(gpu_ctx, width):
    w, h, spp = 640, 480, 8
    ds, cam = gpu_ctx.upload(P.cornell_ref(True)), P.cornell_ref_camera(w, h)
    want, ms = _render(gpu_ctx, ds, cam, w, h, spp, width, 0)
    for block in (1, 32, 64, 96, 160, 256, 1000):
        got, t = _render(gpu_ctx, ds, cam, w, h, spp, width, block)
        np.testing.assert_array_equal(got, want, err_msg=str(block))
        assert t < 1.25 * ms, (block, t, ms)
    ds.close()
