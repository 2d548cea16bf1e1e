"""NEE slots keep what an earlier vertex, or an earlier and deeper call, left in
them: a path adds a slot only for the vertex right after the one that filled it,
or at its end. Films follow the oracle's at every depth after a deeper render,
batch jobs of different depths hold the single renders' bits, and gradients after
a deeper replay are those of a first call."""
import numpy as np
import pytest

from pyre_gb300 import presets as P
from pyre_gb300.scene import CudaIntegrator, DiffuseAreaQuadLight, DisneyBsdf, PathIntegrator

pytestmark = pytest.mark.gpu

W, H, SPP = 40, 30, 4


def _scene(quads, env=True):
    sc = P.studio_ref(True)
    sc.materials[0] = DisneyBsdf([0.6, 0.5, 0.4], 0.3, 0.5, 0.5)
    sc.lights = [DiffuseAreaQuadLight((-0.6 + 0.02 * k, 1.6, -0.3), (0.4, 0, 0), (0, 0, 0.4), (6.0 / quads, 0.3, 0.2))
                 for k in range(quads)]
    if not env:
        sc.env = None
    return sc, P.studio_ref_camera(W, H)


@pytest.mark.parametrize("quads,env", [(0, True), (1, False), (3, True), (40, True)])
@pytest.mark.parametrize("staged", [False, True])
def test_films_after_a_deeper_render(gpu_ctx, oracle_mod, quads, env, staged):
    sc, cam = _scene(quads, env)
    ds, osc = gpu_ctx.upload(sc), oracle_mod.OracleScene(sc)
    gpu_ctx.set_stage_timing(staged)  # timed stages are launches of their own
    gpu_ctx.render(ds, cam, PathIntegrator(9, 9), W, H, SPP)
    for depth in (0, 1, 2, 5):
        got = gpu_ctx.render(ds, cam, PathIntegrator(depth, 2), W, H, SPP, env_sampling=1)
        want = osc.render(cam, W, H, SPP, max_depth=depth, min_rr_depth=2)
        # the same random numbers on both sides: pixels agree but for a path that a transcendental's last bit diverts
        close = np.isclose(got.radiance, want["radiance"], rtol=1e-4, atol=1e-5).all(-1)
        assert close.mean() > 0.97, depth
    gpu_ctx.set_stage_timing(False)
    ds.close()


def test_batch_jobs_of_different_depths(gpu_ctx):
    sc, cam = _scene(3, False)
    ds, bs = gpu_ctx.upload(sc), gpu_ctx.upload_batch([sc])
    depths = [7, 0, 1, 3, 0, 12, 2]
    jobs = [dict(part=0, camera=cam, width=W, height=H, spp=SPP, integrator=PathIntegrator(d, 2)) for d in depths]
    for wave in (0, 2 * W * H):
        for d, film in zip(depths, gpu_ctx.render_batch(bs, jobs, wave_paths=wave)):
            one = gpu_ctx.render(ds, cam, PathIntegrator(d, 2), W, H, SPP)
            np.testing.assert_array_equal(film.radiance, one.radiance, err_msg=str(d))
    bs.close()
    ds.close()


@pytest.mark.parametrize("quads,env", [(0, True), (3, True)])
def test_gradients_after_a_deeper_replay(quads, env):
    sc, cam = _scene(quads, env)
    dl = np.random.default_rng(3).random((H, W, 3)).astype(np.float32)

    def grads(ctx, ds, depth):
        it = PathIntegrator(depth, 2)
        ctx.forward(ds, cam, it, W, H, SPP)
        return ctx.backward(ds, cam, it, W, H, SPP, dl)

    used = CudaIntegrator(0)
    used_ds = used.upload(sc)
    for depth in (0, 1, 2, 4):
        grads(used, used_ds, 9)
        mat, tex = grads(used, used_ds, depth)
        new = CudaIntegrator(0)
        new_ds = new.upload(sc)
        mat0, tex0 = grads(new, new_ds, depth)
        assert depth > 0 or not mat.any()
        assert depth == 0 or mat.any()
        # FP64 sums (materials) and FP32 ones (texels) in any order of their terms
        np.testing.assert_allclose(mat, mat0, rtol=0, atol=1e-10 * max(1.0, np.abs(mat0).max()))
        np.testing.assert_allclose(tex, tex0, rtol=0, atol=1e-4 * max(1e-6, np.abs(tex0).max()))
        new_ds.close()
        new.close()
    used_ds.close()
    used.close()
