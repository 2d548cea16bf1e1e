"""A static instance is found in the same order, and at about the same cost,
whether or not other instances use its mesh: 512 spheres on a grid against the
same spheres whose meshes each have a second, moving user far from every ray.
Hits keep their bits. The twins double the instances but are culled near the
top, so closest-hit and any-hit queries may take a few per cent longer; 15 % is
where entering each sphere the slow way (out of the step loop, box tested twice,
order fixed) begins: it costs a quarter."""
import ctypes as C
import math

import numpy as np
import pytest

from pyre_gb300 import native as N
from pyre_gb300 import presets as P
from pyre_gb300.scene import InstanceMotion, Lambertian, MeshInstance, Primitive, Scene

pytestmark = pytest.mark.gpu

K = 8
RAYS = 1 << 21


def _field(twins):
    sc = Scene()
    sc.materials.append(Lambertian([0.5] * 3))
    away = InstanceMotion((1000.0, 1000.0, 1000.0), (1000.0, 1000.0, 1000.0))
    meshes = [P.make_uv_sphere((2 * i - K + 1, 2 * j - K + 1, 2 * k - K + 1), 0.8, 24, 12)
              for i in range(K) for j in range(K) for k in range(K)]
    sc.primitives = [Primitive(MeshInstance.build(m), 0) for m in meshes]
    if twins:
        sc.primitives += [Primitive(MeshInstance.build_animated(m, away), 0) for m in meshes]
    return sc


def _queries(ctx, ds, rays):
    import torch
    ints = {k: torch.zeros(RAYS, dtype=torch.int32, device="cuda") for k in ("kind", "instance", "triangle")}
    floats = {k: torch.zeros(RAYS, device="cuda") for k in ("t", "u", "v")}
    occ = torch.zeros(RAYS, dtype=torch.uint8, device="cuda")
    desc = N.Rays(*[N.dptr(x) for x in rays])
    hits = N.Hits(*[N.dptr(x, C.c_int32) for x in ints.values()], *[N.dptr(x) for x in floats.values()])
    ms = {"closest": [], "any": []}
    for _ in range(9):
        ctx.check(ctx.lib.pyre_intersect_closest(ctx.handle, ds.handle, C.byref(desc), RAYS, C.byref(hits),
                                                 N.PYRE_MEM_DEVICE))
        ms["closest"].append(ctx.stats().ms_total)
        ctx.check(ctx.lib.pyre_intersect_any(ctx.handle, ds.handle, C.byref(desc), RAYS, N.dptr(occ, C.c_uint8),
                                             N.PYRE_MEM_DEVICE))
        ms["any"].append(ctx.stats().ms_total)
    out = {k: v.cpu().numpy() for k, v in {**ints, **floats, "occluded": occ}.items()}
    return {k: min(v[2:]) for k, v in ms.items()}, out


def test_static_users_of_a_shared_mesh(gpu_ctx):
    import torch
    g = torch.Generator(device="cuda").manual_seed(7)
    org = (torch.rand(RAYS, 3, device="cuda", generator=g) * 2 - 1) * float(K)
    d = torch.randn(RAYS, 3, device="cuda", generator=g)
    rays = (org.contiguous(), (d / d.norm(dim=1, keepdim=True)).contiguous(), torch.full((RAYS,), 1e-4, device="cuda"),
            torch.full((RAYS,), math.inf, device="cuda"), torch.rand(RAYS, device="cuda", generator=g))
    ms, out = {}, {}
    for twins in (False, True):
        ds = gpu_ctx.upload(_field(twins))
        ms[twins], out[twins] = _queries(gpu_ctx, ds, rays)
        ds.close()
    assert (out[False]["kind"] > 0).mean() > 0.5
    away = out[True]["instance"] >= K ** 3  # a ray that passes every sphere may meet a twin far behind them
    assert away.sum() < 100 and not out[False]["kind"][away].any()
    for k, v in out[False].items():
        np.testing.assert_array_equal(v[~away], out[True][k][~away], err_msg=k)
    for k in ("closest", "any"):
        assert ms[True][k] < 1.15 * ms[False][k], (k, ms)
