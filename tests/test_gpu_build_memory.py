"""What the GPU BVH build leaves on the device: a context keeps at most 512 MiB
of its workspace between builds of a mesh, 16 MiB after a scene upload, and
gives it back when another allocation finds the device full."""
import numpy as np
import pytest

from pyre_gb300 import presets as P
from pyre_gb300.native import PyreError
from pyre_gb300.scene import CudaIntegrator, PathIntegrator, TriangleMesh

pytestmark = pytest.mark.gpu

KEPT = 512 << 20
UPLOAD = 16 << 20
SLACK = 8 << 20  # granularity of the driver's allocations


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info(0)[0]


def _builder():
    ctx = CudaIntegrator(0)
    ctx.set_bvh_builder("device")
    ctx.bvh_build(P.icosphere_displaced(2, 0.1))  # loads the kernels; their memory stays
    return ctx


def _grid(n):
    """2 n^2 triangles of a height field."""
    rng = np.random.default_rng(n)
    x, z = np.meshgrid(np.arange(n + 1, dtype=np.float32), np.arange(n + 1, dtype=np.float32), indexing="ij")
    pos = np.stack([x, rng.random(x.shape, dtype=np.float32), z], -1).reshape(-1, 3)
    a = (np.arange(n)[:, None] * (n + 1) + np.arange(n)).astype(np.uint32)
    idx = np.stack([a, a + 1, a + n + 1, a + 1, a + n + 2, a + n + 1], -1)
    return TriangleMesh(pos, idx.reshape(-1))


@pytest.mark.parametrize("n,kept", [(30, True), (380, True), (1000, False)])
def test_build_workspace_is_bounded(n, kept):
    ctx = _builder()
    mesh = _grid(n)
    before = _free()
    nodes, prim = ctx.bvh_build(mesh)
    assert before - _free() <= (KEPT if kept else 0) + SLACK
    again = ctx.bvh_build(mesh)
    np.testing.assert_array_equal(nodes, again[0])
    np.testing.assert_array_equal(prim, again[1])
    ctx.close()


def test_a_full_device_gets_the_workspace_back():
    ctx = _builder()
    sc, cam = P.cornell_box(), P.cornell_box_camera(16, 16)
    ds = ctx.upload(sc)
    film = ctx.render(ds, cam, PathIntegrator(3, 2), 16, 16, 1)
    ctx.set_bvh_builder("host")
    before = _free()
    ctx.bvh_build(_grid(380))
    assert before - _free() > 64 << 20
    with pytest.raises(PyreError, match="cudaMalloc"):  # keeps 16 bytes of each of 2^37 paths: more than any device has
        ctx.forward(ds, cam, PathIntegrator(3, 2), 16, 16, 1 << 29)
    assert before - _free() <= SLACK
    again = ctx.render(ds, cam, PathIntegrator(3, 2), 16, 16, 1)
    np.testing.assert_array_equal(film.radiance, again.radiance)
    nodes, _ = ctx.bvh_build(_grid(30))
    assert len(nodes) > 1
    ds.close()
    ctx.close()


def test_upload_gives_the_workspace_back():
    ctx = _builder()
    sc = P.microbench_scene(7)
    small = P.cornell_box()
    ctx.upload(small).close()
    before = _free()
    ds = ctx.upload(sc)
    info = ds.info()
    assert before - _free() <= info.device_bytes + SLACK + UPLOAD
    ds.close()
    assert before - _free() <= SLACK + UPLOAD
    ctx.render(ctx.upload(small), P.cornell_box_camera(16, 16), PathIntegrator(3, 2), 16, 16, 1)
    ctx.close()
