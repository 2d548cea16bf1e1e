"""Captured waves: a render that replays a graph gives the bits and the launch
counts of the same render without one, whatever was captured before it. Crops
of one area but of different shape or place, and launch shapes that differ only
in whether a small wave runs as one launch, need a graph of their own."""
import numpy as np
import pytest

from pyre_gb300 import native as N
from pyre_gb300 import presets as P
from pyre_gb300.scene import Film, PathIntegrator

pytestmark = pytest.mark.gpu


def _render(ctx, ds, cam, w, h, crop, graph, **knobs):
    film = Film(crop[2] - crop[0], crop[3] - crop[1])
    f = N.Film(N.fptr(film.radiance), N.fptr(film.albedo), N.fptr(film.normal), N.fptr(film.depth), N.PYRE_MEM_HOST)
    ctx.render_into(ds, cam, ctx.params(w, h, 3, 6, PathIntegrator(5, 2), crop=crop, use_graph=graph, **knobs), f)
    return film, ctx.stats().kernel_launches


def _check(ctx, w, h, steps):
    ds, cam = ctx.upload(P.cornell_ref(True)), P.cornell_ref_camera(w, h)
    plain = [_render(ctx, ds, cam, w, h, crop, 0, **knobs) for crop, knobs in steps]
    graph = [_render(ctx, ds, cam, w, h, crop, 1, **knobs) for crop, knobs in steps]
    ds.close()
    for (a, launches_a), (b, launches_b), step in zip(plain, graph, steps):
        assert launches_a == launches_b, step
        for k in ("radiance", "albedo", "normal", "depth"):
            np.testing.assert_array_equal(getattr(b, k), getattr(a, k), err_msg=f"{step} {k}")


def test_crops_of_one_area(gpu_ctx):
    _check(gpu_ctx, 64, 48, [((0, 0, 32, 16), {}), ((0, 0, 16, 32), {}), ((0, 0, 64, 8), {}), ((16, 0, 32, 32), {}),
                             ((0, 16, 16, 48), {}), ((0, 0, 32, 16), {})])


def test_crop_origins_far_apart(gpu_ctx):
    _check(gpu_ctx, 65600, 2, [((65536, 0, 65568, 1), {}), ((0, 1, 32, 2), {})])


def test_one_launch_and_staged_waves(gpu_ctx):
    crop = (0, 0, 64, 48)
    _check(gpu_ctx, 64, 48, [(crop, {}), (crop, {"block_size": 256}), (crop, {}), (crop, {"block_size": 128}),
                             (crop, {"refill_lanes": 12}), (crop, {"wave_paths": 64 * 48})])
