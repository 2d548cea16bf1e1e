"""The radiance kept for the adjoint belongs to the scene's parameters at the
time: after new materials or a new environment, pyre_backward without another
pyre_forward gives the gradients of the new parameters, those of a context that
never saw the old ones."""
import numpy as np
import pytest

from pyre_gb300 import presets as P
from pyre_gb300.scene import CudaIntegrator, DisneyBsdf, Lambertian, PathIntegrator

pytestmark = pytest.mark.gpu

W, H, SPP = 40, 30, 4
IT = PathIntegrator(5, 2)


def _changed(materials):
    return [Lambertian(np.clip(0.5 * m.albedo + 0.2, 0, 1)) if isinstance(m, Lambertian)
            else DisneyBsdf(np.clip(0.5 * np.asarray(m.base_color) + 0.2, 0, 1), 0.3, 0.6, 0.4) for m in materials]


@pytest.mark.parametrize("what", ["materials", "env"])
@pytest.mark.parametrize("first", ["forward", "backward"])
def test_gradients_after_a_change_without_forward(gpu_ctx, what, first):
    sc, cam = P.adjoint_check_scene()
    dl = np.random.default_rng(4).random((H, W, 3)).astype(np.float32)
    ds = gpu_ctx.upload(sc)
    if first == "forward":
        gpu_ctx.forward(ds, cam, IT, W, H, SPP)
    else:
        gpu_ctx.backward(ds, cam, IT, W, H, SPP, dl)
    if what == "materials":
        gpu_ctx.set_materials(ds, _changed(sc.materials))
    else:
        gpu_ctx.set_env(ds, sc.env.pixels * np.float32(0.25) + np.float32(0.5), 2.0)
    mat, env = gpu_ctx.backward(ds, cam, IT, W, H, SPP, dl)
    changed = ds.scene
    ds.close()
    fresh = CudaIntegrator(0)
    fds = fresh.upload(changed)
    mat0, env0 = fresh.backward(fds, cam, IT, W, H, SPP, dl)
    fds.close()
    fresh.close()
    assert mat0.any() and env0.any()
    # FP64 sums (materials) and FP32 ones (texels) of the same terms in any order
    np.testing.assert_allclose(mat, mat0, rtol=0, atol=1e-10 * np.abs(mat0).max())
    np.testing.assert_allclose(env, env0, rtol=0, atol=1e-4 * np.abs(env0).max())

