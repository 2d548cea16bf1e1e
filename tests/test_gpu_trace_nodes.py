"""The forms a scene's traversal nodes can take: static instances hung below the
top level, instances entered at their root box (moving, or of a mesh that
several instances use), top-level leaves of several instances, one-leaf BVHs
with an empty second child. Hits equal the oracle's bit for bit."""
import numpy as np
import pytest

from pyre_gb300 import presets as P
from pyre_gb300.scene import InstanceMotion, Lambertian, MeshInstance, Primitive, Scene, TriangleMesh

pytestmark = pytest.mark.gpu


def _scene(name):
    sc = Scene()
    sc.materials.append(Lambertian([0.5] * 3))
    ball = P.make_uv_sphere((0.0, 0.0, 0.0), 0.5, 16, 8)
    tri = TriangleMesh(np.float32([[-1, -1, 0], [1, -1, 0], [0, 1, 0]]), np.uint32([0, 1, 2]))
    quad = P.quad_mesh([(-2, -0.5, -2), (2, -0.5, -2), (2, -0.5, 2), (-2, -0.5, 2)], (0, 1, 0))
    move = InstanceMotion((0, 0, 0), (0.4, 0.2, -0.3))
    rest = InstanceMotion((0, 0, 0), (0, 0, 0))

    def add(mesh, motion=None):
        inst = MeshInstance.build(mesh) if motion is None else MeshInstance.build_animated(mesh, motion)
        sc.primitives.append(Primitive(inst, 0))

    for mesh, motion in {
        "one-triangle": [(tri, None)],
        "shared-static": [(ball, None), (quad, None), (ball, None)],            # coincident: ties, one top-level leaf
        "shared-static-moving": [(ball, None), (ball, move), (quad, None), (tri, None)],
        "all-moving": [(ball, move), (tri, rest), (quad, move)],
        "mixed": [(quad, None), (ball, move), (tri, None), (P.make_uv_sphere((1.2, 0.1, 0.3), 0.4, 8, 4), None),
                  (P.make_uv_sphere((-1.2, 0.1, 0.3), 0.4, 8, 4), rest)],
        "same-centroid": [(P.make_uv_sphere((0, 0, 0), r, 8, 4), None) for r in (0.2, 0.4, 0.6, 0.8)],
    }[name]:
        add(mesh, motion)
    return sc


@pytest.mark.parametrize("width", [2, 4, 8])
@pytest.mark.parametrize("name", ["one-triangle", "shared-static", "shared-static-moving", "all-moving", "mixed",
                                  "same-centroid"])
def test_node_forms_match_the_oracle(gpu_ctx, oracle_mod, name, width):
    sc = _scene(name)
    rng = np.random.default_rng(3)
    n = 20_000
    org = (rng.random((n, 3)) * 4 - 2).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    # along the diagonal of an empty child's box, and along the axes with signed zeros
    d[:64] = np.float32([1, 2, 4])
    d[64:128] = np.float32([-1, -2, -4])
    d[128:256] = np.float32([[0.0, -0.0, 1.0], [-0.0, 0.0, -1.0], [1.0, 0.0, -0.0], [0.0, -1.0, 0.0]] * 32)
    tmin = np.full(n, 1e-4, np.float32)
    tmax = np.where(rng.random(n) < 0.5, np.inf, rng.random(n) * 3).astype(np.float32)
    time = rng.random(n).astype(np.float32)
    ref = oracle_mod.OracleScene(sc)
    ds = gpu_ctx.upload(sc)
    ds.set_bvh_width(width)
    got, want = gpu_ctx.intersect(ds, org, d, tmin, tmax, time=time), ref.intersect(org, d, tmin, tmax, time=time)
    for k in ("kind", "instance", "triangle"):
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    hit = want["kind"] > 0
    for k in ("t", "u", "v"):
        np.testing.assert_array_equal(got[k][hit].view(np.uint32), want[k][hit].view(np.uint32), err_msg=k)
    occ = gpu_ctx.intersect(ds, org, d, tmin, tmax, time=time, any_hit=True)
    np.testing.assert_array_equal(occ, ref.occluded(org, d, tmin, tmax, time=time))
    ds.close()
