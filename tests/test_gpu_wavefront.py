"""Wavefront shapes of the path tracer: bounces over the live paths only, and
the launch that follows the last paths to their ends, which starts once they
fit the chip at once (152 x 8 blocks of 128)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(a, b):
    """One sample per pixel: the same terms in the same order, so a pixel may
    differ by the rounding of about 50 operations (50 x 2^-24 = 3e-6, taken
    twice), except where a last-bit difference flips a choice of the path."""
    close = np.isclose(a, b, rtol=6e-6, atol=1e-7).all(axis=-1)
    assert close.mean() >= 0.999, close.mean()


@pytest.mark.parametrize("integrator", ["path", "path_filtered_ss"])
@pytest.mark.parametrize("size, max_paths", [((1, 1), 0), ((43, 3), 127), ((43, 3), 128), ((43, 3), 129),
                                             ((480, 330), 1000), ((480, 330), 157000)])
def test_live_paths_and_finish(sms, workloads, gpu_lib, integrator, size, max_paths):
    """480 x 330 paths are more than the chip holds: bounces at first, the
    finishing launch later; smaller wavefronts take it from the camera on."""
    W = workloads
    ctx = sms.Context(sms.Scene(W.pool_scene(res=32)), W.water_config())
    cam = W.pool_camera(*size)
    full = ctx.render(cam, sms.RenderOptions(integrator=integrator, spp=1, seed=9))
    part = ctx.render(cam, sms.RenderOptions(integrator=integrator, spp=1, seed=9, max_paths=max_paths))
    again = ctx.render(cam, sms.RenderOptions(integrator=integrator, spp=1, seed=9))
    ctx.close()
    assert np.array_equal(full, again)
    _same(full, part)


def test_render_buffers_are_kept_and_shared(sms, workloads, gpu_lib):
    """A context's render buffers serve images of any size and integrator in
    any order, and two threads at a time: every image equals a new context's."""
    import threading
    W = workloads
    desc, cfg = W.pool_scene(res=32), W.water_config()
    jobs = [(7, 5, "path_sms_ss", 1), (120, 90, "path", 2), (16, 16, "path_sms_ss", 2), (50, 2, "path", 1)]
    opt = {j: sms.RenderOptions(integrator=j[2], spp=j[3], seed=2) for j in jobs}
    want = {}
    for j in jobs:
        ctx = sms.Context(sms.Scene(desc), cfg)
        want[j] = ctx.render(W.pool_camera(*j[:2]), opt[j])
        ctx.close()
    ctx = sms.Context(sms.Scene(desc), cfg)
    for j in jobs + jobs[::-1]:
        assert np.array_equal(ctx.render(W.pool_camera(*j[:2]), opt[j]), want[j]), j
    got = {}

    def work(j):
        got[j] = [ctx.render(W.pool_camera(*j[:2]), opt[j]) for _ in range(4)]

    threads = [threading.Thread(target=work, args=(j,)) for j in jobs if j[2] == "path"]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=60)
    ctx.close()
    for j, images in got.items():
        for img in images:
            assert np.array_equal(img, want[j]), j
    assert len(got) == 2
