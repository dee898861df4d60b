"""The biased single-scatter estimator on both sides of the batch size from which
its kernel is compiled for more blocks per SM (8 blocks of 128 walks per SM for
smooth casters, 32 for two-stage normal-mapped ones; 152 SMs): a large batch
gives every query the result it has in a small one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind, n, trials", [("water", 4864, 32), ("water", 4868, 32), ("water", 9737, 16),
                                             ("pane", 19456, 17), ("pane", 19460, 17)])
def test_large_batches_equal_small_ones(sms, workloads, gpu_lib, kind, n, trials):
    W = workloads
    if kind == "water":
        desc, cfg = W.water_scene(res=32), sms.SMSConfig(biased=True, max_trials=trials)
    else:
        desc = W.nm_plane_scene(conductor=False, res=64)
        cfg = sms.SMSConfig(biased=True, max_trials=trials, twostage=True)
    rng = np.random.default_rng(n)
    q = W.plane_queries(rng.uniform(-0.5, 0.5, (n, 2)).astype(np.float32))
    ctx = sms.Context(sms.Scene(desc), cfg)
    ss = sms.SpecularManifoldSingleScatter(ctx)
    value, count, walks = ss.specular_manifold_sampling(q, seed=4)
    for a in range(0, n, 2400):
        b = min(n, a + 2400)
        v, c, w = ss.specular_manifold_sampling(np.ascontiguousarray(q[:, a:b]), seed=4, stream_offset=a)
        assert np.array_equal(c, count[a:b]) and np.array_equal(w, walks[a:b])
        # contributions: the rounding of about 100 operations
        np.testing.assert_allclose(v, value[:, a:b], rtol=1e-5, atol=1e-9)
    ctx.close()
