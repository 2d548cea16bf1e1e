"""Waves that run as one launch against the same render stage by stage (a
block_size keeps a render on the stage kernels): every channel's bits, and the
ray counts, for slices of one path, ragged slices, both sides of the limit,
several waves, and each kind of light."""
import numpy as np
import pytest

from pyre_gb300 import native as N
from pyre_gb300 import presets as P
from pyre_gb300.scene import DiffuseAreaQuadLight, Film, PathIntegrator

pytestmark = pytest.mark.gpu


def _scene(name):
    if name == "quads":
        return P.cornell_ref(True), P.cornell_ref_camera
    sc = P.studio_ref(True)
    if name == "both":
        sc.lights = [DiffuseAreaQuadLight((-0.5, 1.5, -0.3), (0.4, 0, 0), (0, 0, 0.4), (6.0, 5.0, 4.0)),
                     DiffuseAreaQuadLight((0.3, 1.4, -0.2), (0.2, 0, 0), (0, 0, 0.2), (3.0, 5.0, 8.0))]
    elif name == "none":
        sc.env = None
    return sc, lambda w, h: P.studio_ref_camera(w, h, aperture=0.05)


def _render(ctx, ds, cam, it, w, h, spp, **knobs):
    film = Film(w, h)
    f = N.Film(N.fptr(film.radiance), N.fptr(film.albedo), N.fptr(film.normal), N.fptr(film.depth), N.PYRE_MEM_HOST)
    ctx.render_into(ds, cam, ctx.params(w, h, 5, 5 + spp, it, **knobs), f)
    s = ctx.stats()
    return film, (s.samples, s.extend_rays, s.shadow_rays), s.kernel_launches


@pytest.mark.parametrize("name", ["quads", "env", "both", "none"])
@pytest.mark.parametrize("w,h,spp,depth,wave", [(1, 1, 1, 8, 0), (1, 1, 40, 3, 0), (7, 5, 3, 8, 0), (33, 31, 1, 1, 0),
                                                (64, 64, 32, 8, 0), (64, 64, 33, 8, 0), (61, 47, 11, 12, 9000)])
def test_one_launch_equals_the_stages(gpu_ctx, name, w, h, spp, depth, wave):
    sc, camera = _scene(name)
    ds, cam, it = gpu_ctx.upload(sc), camera(w, h), PathIntegrator(depth, 2)
    one, rays_one, launches = _render(gpu_ctx, ds, cam, it, w, h, spp, wave_paths=wave)
    ref, rays_ref, staged = _render(gpu_ctx, ds, cam, it, w, h, spp, wave_paths=wave, block_size=256)
    ds.close()
    assert rays_one == rays_ref
    assert launches < staged or w * h * spp > 128 * 1024 or depth == 1
    for k in ("radiance", "albedo", "normal", "depth"):
        np.testing.assert_array_equal(getattr(one, k), getattr(ref, k), err_msg=k)
