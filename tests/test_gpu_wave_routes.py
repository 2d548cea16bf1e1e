"""What a wave launches, on both sides of the one-launch limit, through every
entry point that renders one: the reported launches are those of the route that
ran, and the film's bits are those of the timed stages, which are always
launches of their own."""
import ctypes as C

import numpy as np
import pytest

from pyre_gb300 import native as N
from pyre_gb300 import presets as P
from pyre_gb300.scene import CudaIntegrator, PathIntegrator

pytestmark = pytest.mark.gpu

LIMIT = 128 * 1024  # paths of the largest wave that runs as one launch


def _staged(depth, timed):
    """begin, raygen, accumulate, end; shade per depth; extend at depth 0, then shadow and extend together or apart."""
    return 4 + depth + (2 * depth if timed else depth + 1)


def _noalloc(ctx, ds, cam, params, npix):
    import torch
    dev = torch.full((npix * 3,), -1.0, device="cuda")
    film = N.Film(N.dptr(dev), None, None, None, N.PYRE_MEM_DEVICE)
    desc = cam.to_desc()
    ctx.check(ctx.lib.pyre_render_noalloc(ctx.handle, ds.handle, C.byref(desc), C.byref(params), C.byref(film)))
    return dev.cpu().numpy()


@pytest.mark.parametrize("w,h,spp,depth", [(16, 9, 2, 1), (16, 9, 2, 7), (64, 64, 32, 1), (64, 64, 32, 6),
                                           (64, 64, 33, 1), (64, 64, 33, 6)])
@pytest.mark.parametrize("timing", [False, True])
def test_launch_counts(gpu_ctx, w, h, spp, depth, timing):
    sc, cam, it = P.cornell_ref(True), P.cornell_ref_camera(w, h), PathIntegrator(depth, 2)
    ds = gpu_ctx.upload(sc)
    gpu_ctx.set_stage_timing(True)
    ref = gpu_ctx.render(ds, cam, it, w, h, spp)
    assert gpu_ctx.stats().kernel_launches == _staged(depth, True) + 1
    gpu_ctx.set_stage_timing(timing)
    one = 4 if w * h * spp <= LIMIT else _staged(depth, False)
    for graph in (0, 1):
        got = gpu_ctx.render(ds, cam, it, w, h, spp, use_graph=graph)
        assert gpu_ctx.stats().kernel_launches == (_staged(depth, True) if timing else one) + 1
        np.testing.assert_array_equal(got.radiance, ref.radiance)
    # without allocations: stages are never timed; the static array holds each of these waves whole
    rad = _noalloc(gpu_ctx, ds, cam, CudaIntegrator.params(w, h, 0, spp, it), w * h)
    s = gpu_ctx.stats()
    np.testing.assert_array_equal(rad.reshape(ref.radiance.shape), ref.radiance)
    assert s.waves == 1 and s.kernel_launches == one + 1
    gpu_ctx.set_stage_timing(False)
    ds.close()


@pytest.mark.parametrize("w,h,passes", [(17, 5, 3), (64, 64, 32), (64, 64, 33)])
def test_progressive_passes(gpu_ctx, w, h, passes):
    sc, cam, it = P.studio_ref(True), P.studio_ref_camera(w, h, aperture=0.05), PathIntegrator(6, 2)
    ds = gpu_ctx.upload(sc)
    got = gpu_ctx.render_progressive(ds, cam, it, w, h, passes)
    assert gpu_ctx.stats().kernel_launches == (4 if w * h * passes <= LIMIT else _staged(6, False)) + 1
    want = gpu_ctx.render_progressive(ds, cam, it, w, h, passes, block_size=256)
    assert gpu_ctx.stats().kernel_launches == _staged(6, False) + 1
    np.testing.assert_array_equal(got, want)
    ds.close()
