"""GPU BVH build at the sizes where its passes change hands: ranges of 32 and 33
primitives (finished by one warp or split by the level kernels), 512 positions
per block, 4096 per scan block, and uploads of meshes on both sides of them.
Node for node equal to the host build."""
import numpy as np
import pytest

from pyre_gb300.scene import Lambertian, MeshInstance, Primitive, Scene, TriangleMesh, build_bvh

pytestmark = pytest.mark.gpu


def _mesh(n, shape, seed=0):
    rng = np.random.default_rng(seed + n)
    pos = rng.uniform(-1, 1, (3 * n, 3)).astype(np.float32)
    if shape == "coincident":
        pos[:] = np.tile(np.float32([[0, 0, 0], [1, 0, 0], [0, 1, 0]]), (n, 1))
    elif shape == "planar":
        pos[:, 1] = 0.0
    elif shape == "clusters":  # runs of equal centroids beside spread ones
        pos = (np.repeat(rng.integers(0, 3, n), 3)[:, None] * 2 + np.tile(np.float32([[0, 0, 0], [.5, 0, 0], [0, .5, .5]]), (n, 1)))
        pos[: 3 * (n // 2)] += rng.uniform(-.1, .1, (3 * (n // 2), 3))
    return TriangleMesh(pos.astype(np.float32), np.arange(3 * n, dtype=np.uint32))


@pytest.mark.parametrize("shape", ["soup", "coincident", "planar", "clusters"])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 34, 65, 511, 512, 513, 1025, 4095, 4096, 4097, 20_000])
def test_sizes_at_the_edges(gpu_ctx, n, shape):
    mesh = _mesh(n, shape)
    want_nodes, want_prim = build_bvh(mesh)
    nodes, prim = gpu_ctx.bvh_build(mesh)
    np.testing.assert_array_equal(prim, want_prim)
    assert len(nodes) == len(want_nodes)
    for k in nodes.dtype.names:
        np.testing.assert_array_equal(nodes[k], want_nodes[k], err_msg=k)


def test_upload_of_small_and_large_meshes(gpu_ctx):
    sc = Scene()
    sc.materials.append(Lambertian([0.5] * 3))
    for k, n in enumerate((1, 33, 7, 600, 32, 2, 4100)):
        m = _mesh(n, "soup", seed=k)
        m.positions[:] = m.positions * 0.3 + np.float32([k - 3, 0, 0])
        sc.primitives.append(Primitive(MeshInstance.build(m), 0))
    rng = np.random.default_rng(1)
    org = rng.uniform(-4, 4, (50_000, 3)).astype(np.float32)
    d = rng.normal(size=(50_000, 3)).astype(np.float32)
    tmin, tmax = np.full(50_000, 1e-4, np.float32), np.full(50_000, np.inf, np.float32)
    got = {}
    for builder in ("host", "device"):
        gpu_ctx.set_bvh_builder(builder)
        ds = gpu_ctx.upload(sc)
        got[builder] = gpu_ctx.intersect(ds, org, d, tmin, tmax)
        ds.close()
    gpu_ctx.set_bvh_builder("host")
    assert (got["host"]["kind"] > 0).any()
    for k, v in got["host"].items():
        np.testing.assert_array_equal(got["device"][k], v, err_msg=k)
