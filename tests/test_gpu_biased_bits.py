"""The biased single-scatter estimator gives a query the same bits in a large
batch, whose kernel is compiled for more blocks per SM, as in a small one:
splitting a batch with stream_offset keeps results identical."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# blocks of 128 lanes per SM from which a batch is large, and lanes a query
@pytest.mark.parametrize("kind, large, lanes", [("water", 8, 32), ("water", 8, 16), ("sphere", 8, 32), ("pane", 32, 32),
                                                ("pane", 32, 16)])
@pytest.mark.parametrize("past", [0, 1])
def test_large_batches_are_the_same_bits(sms, workloads, gpu_lib, kind, large, lanes, past):
    import torch
    W = workloads
    sms_count = torch.cuda.get_device_properties(0).multi_processor_count
    per_block = 128 // lanes
    n = per_block * (large * sms_count + past)   # the last small batch, the first large one
    opts = dict(biased=True, max_trials=32 if lanes == 32 else 16)
    if kind == "pane":
        desc, cfg = W.nm_plane_scene(conductor=False, res=64), sms.SMSConfig(twostage=True, **opts)
    else:
        desc = W.water_scene(res=32) if kind == "water" else W.sphere_scene(conductor=True)
        cfg = sms.SMSConfig(**opts)
    rng = np.random.default_rng(n)
    extent = 2.0 if kind == "sphere" else 1.0   # the sphere's reflections fall beside it
    q = W.plane_queries(rng.uniform(-extent, extent, (n, 2)).astype(np.float32))
    ctx = sms.Context(sms.Scene(desc), cfg)
    ss = sms.SpecularManifoldSingleScatter(ctx)
    whole = ss.specular_manifold_sampling(q, seed=4)
    assert (whole[1] > 0).any()
    for a in range(0, n, 2400):
        b = min(n, a + 2400)
        part = ss.specular_manifold_sampling(np.ascontiguousarray(q[:, a:b]), seed=4, stream_offset=a)
        for x, y in zip(whole, part):
            assert np.array_equal(x[..., a:b], y)
    ctx.close()
