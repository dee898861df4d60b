"""Images do not depend on the wavefront size, to the last bit: the launch that
follows the last paths of a query-free integrator to their ends gives the paths
what the bounce launches give them.  One sample per pixel, so that the order of
a pixel's sum plays no part."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# more paths than a 152-SM chip holds at once (155,648): the default wavefront
# starts with bounce launches, the small ones finish from the camera on
SIZE = (480, 330)


def _spheres(sms, W):
    """A mirror and a glass sphere over a floor under a sphere light; no radius
    is a power of two."""
    d = sms.SceneDesc()
    P = np.array([[-2, -2, 0], [2, -2, 0], [2, 2, 0], [-2, 2, 0]], np.float32)
    uv = np.array([[0, 0], [1, 0], [1, 1], [0, 1]], np.float32)
    d.add_mesh(P, np.array([[0, 1, 2], [0, 2, 3]], np.uint32), sms.Bsdf(sms.BSDF_DIFFUSE, 1.0, 0.0, (0.5,) * 3),
               sms.SHAPE_CAUSTIC_RECEIVER, UV=uv)
    d.add_sphere((-0.7, 0.0, 0.8), 0.35, sms.Bsdf(sms.BSDF_CONDUCTOR, 0.2, 3.0), sms.SHAPE_CAUSTIC_CASTER_SINGLE)
    d.add_sphere((0.6, 0.3, 0.7), 0.37, sms.Bsdf(sms.BSDF_DIELECTRIC, 1.5), sms.SHAPE_CAUSTIC_CASTER_SINGLE)
    light = d.add_sphere((0.0, 0.5, 4.0), 0.43, sms.Bsdf(sms.BSDF_DIFFUSE, 1.0, 0.0, (0.0,) * 3), 0)
    d.add_area_emitter(light, (40.0,) * 3, sms.EMITTER_CAUSTIC_SINGLE | sms.EMITTER_CAUSTIC_MULTI)
    return d, W.teaser_camera


def _scene(sms, W, name):
    if name == "spheres":
        return _spheres(sms, W)
    if name == "teaser":   # mirror sphere, glass mesh, normal-mapped tile, point light
        return W.teaser_scene(), W.teaser_camera
    return W.pool_scene(res=32), W.pool_camera


@pytest.mark.parametrize("scene", ["spheres", "teaser", "pool"])
@pytest.mark.parametrize("integrator", ["path", "path_filtered_ss", "path_filtered_ms", "path_filtered_teaser"])
def test_wavefront_size_does_not_change_images(sms, workloads, gpu_lib, scene, integrator):
    desc, camera = _scene(sms, workloads, scene)
    ctx = sms.Context(sms.Scene(desc), sms.SMSConfig(max_trials=16, bounces=2))
    cam = camera(*SIZE)
    for seed in (9, 10, 11):
        images = [ctx.render(cam, sms.RenderOptions(integrator=integrator, spp=1, seed=seed, max_depth=12,
                                                    max_paths=m)) for m in (0, 157000, 1000)]
        for m, img in zip((157000, 1000), images[1:]):
            assert np.array_equal(images[0], img), (seed, m, int((images[0] != img).any(axis=-1).sum()))
    ctx.close()
