"""Scheduling of the Bernoulli trials (sms_trials.cuh): the trial counts do not
depend on how many queries a call holds, which decides the lanes per warp, the
number of passes and the claim size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solvers(sms, W):
    """(solver, queries) of each unbiased estimator, on scenes whose walks are
    well conditioned (oracle parity) or whose trial counts vary widely (splits)."""
    glint = W.glint_config()
    glint.biased = glint.glints_vectorized = False
    slab = W.slab_config()
    slab.biased = False
    return {
        "sphere": (sms.SpecularManifoldSingleScatter, W.sphere_scene(conductor=True),
                   sms.SMSConfig(max_trials=512), W.sphere_queries(160)),
        "water": (sms.SpecularManifoldSingleScatter, W.water_scene(res=64), sms.SMSConfig(max_trials=64),
                  W.water_queries(25600)),
        "slab": (sms.SpecularManifoldMultiScatter, W.slab_scene(res=64), slab, W.slab_queries(25600)),
        "glints": (sms.SpecularManifoldGlints, W.glint_scene(map_res=256), glint, W.glint_queries(200)),
    }


@pytest.mark.parametrize("kind", ["sphere", "water", "slab", "glints"])
@pytest.mark.parametrize("sizes", [(1, 2, 31, 33, 1000), (12000, 7)])
def test_batch_size_does_not_change_results(sms, workloads, gpu_lib, kind, sizes):
    cls, desc, cfg, q = _solvers(sms, workloads)[kind]
    ctx = sms.Context(sms.Scene(desc), cfg)
    solver = cls(ctx)
    n = min(q.shape[1], 25600)
    q = np.ascontiguousarray(q[:, :n])
    v, c, w = solver.specular_manifold_sampling(q, seed=5)
    assert (c > 0).any() and (w >= 1).any()
    st = ctx.stats()
    assert st["walks"] == w.sum()
    assert st["bernoulli_trial_iterations_max"] == np.where(c == -1, cfg.max_trials + 1, c).max()
    at = 0
    for k in sizes:
        part = solver.specular_manifold_sampling(np.ascontiguousarray(q[:, at:at + k]), seed=5, stream_offset=at)
        for got, ref in zip(part, (v[:, at:at + k], c[at:at + k], w[at:at + k])):
            assert np.array_equal(got, ref)
        at += k
    ctx.close()


@pytest.mark.parametrize("n", [1, 33, 25600])
@pytest.mark.parametrize("group", [0, 8])
def test_trial_counts_match_the_sequential_oracle(sms, workloads, oracle, gpu_lib, n, group):
    """On the conductor sphere every walk is well conditioned but for 0.1 % (the
    rate the parity tests of the walks allow): counts and walks equal the
    oracle's, which runs the trials one after the other."""
    cls, desc, cfg, q = _solvers(sms, workloads)["sphere"]
    q = np.ascontiguousarray(q[:, (q.shape[1] - n) // 2:][:, :n])
    ctx = sms.Context(sms.Scene(desc), cfg)
    ctx.set_trial_group(group)
    v, c, w = cls(ctx).specular_manifold_sampling(q, seed=9)
    ctx.close()
    vo, co, wo, _ = oracle.OracleScene(desc).connect_batch(cfg, q, seed=9)
    assert np.mean((c != co) | (w != wo)) <= 0.005
    same = c == co
    np.testing.assert_allclose(v[:, same], vo[:, same], rtol=5e-3, atol=1e-7)
