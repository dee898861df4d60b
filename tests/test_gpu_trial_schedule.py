"""Which trials of the stream run when (sms_trials.cuh): nothing of it changes a
result, and calls do not run trials that cannot count."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", ["single", "multi"])
def test_deterministic_seeds_run_no_speculative_trials(sms, workloads, gpu_lib, solver):
    """With mnee_init every trial of a query is its first walk again: the first
    trial decides, and no query has a trial past a success."""
    W = workloads
    if solver == "single":
        desc, cls, q = W.water_scene(res=64), sms.SpecularManifoldSingleScatter, W.water_queries(9000)
        cfg = sms.SMSConfig(max_trials=32, mnee_init=True)
    else:
        desc, cls, q = W.slab_scene(res=64), sms.SpecularManifoldMultiScatter, W.slab_queries(9000)
        cfg = sms.SMSConfig(max_trials=32, mnee_init=True, bounces=2, max_iterations=30)
    ctx = sms.Context(sms.Scene(desc), cfg)
    _, count, walks = cls(ctx).specular_manifold_sampling(q, seed=3)
    st = ctx.stats()
    ctx.close()
    assert (count == 1).sum() > 100 and set(np.unique(count)) <= {-1, 0, 1}
    assert st["walks"] == walks.sum()
    assert st["speculative_walks"] == 0


@pytest.mark.parametrize("n", [52000, 56500, 113000, 130000])
@pytest.mark.parametrize("blocks", [0, 3])
def test_streams_of_one_and_two_grids(sms, workloads, gpu_lib, n, blocks):
    """Streams of half a trial to a few trials a lane of the grid, whose last part
    is shared out: the same results as in small batches."""
    W = workloads
    q = W.water_queries(n)
    ctx = sms.Context(sms.Scene(W.water_scene(res=64)), sms.SMSConfig(max_trials=32))
    ctx.set_launch(blocks, 0)
    ss = sms.SpecularManifoldSingleScatter(ctx)
    whole = ss.specular_manifold_sampling(q, seed=5)
    assert (whole[1] == -1).any() and (whole[1] > 1).any()
    for a in range(0, n, 20000):
        b = min(n, a + 20000)
        part = ss.specular_manifold_sampling(np.ascontiguousarray(q[:, a:b]), seed=5, stream_offset=a)
        for x, y in zip(whole, part):
            assert np.array_equal(x[..., a:b], y)
    ctx.close()


@pytest.mark.parametrize("res", [2, 16, 17, 18])
@pytest.mark.parametrize("n", [1, 305, 2500])
def test_small_trees(sms, workloads, gpu_lib, res, n):
    """Trees around the size from which walks spread over all warps (512
    triangles: 17 x 17 vertices): a query's result is the same alone, in a small
    batch and in a larger one."""
    W = workloads
    q = W.water_queries(5000)
    ctx = sms.Context(sms.Scene(W.water_scene(res=res)), sms.SMSConfig(max_trials=48))
    ss = sms.SpecularManifoldSingleScatter(ctx)
    whole = ss.specular_manifold_sampling(q, seed=8)
    part = ss.specular_manifold_sampling(np.ascontiguousarray(q[:, 40:40 + n]), seed=8, stream_offset=40)
    ctx.close()
    assert (whole[1] > 0).any()
    for x, y in zip(whole, part):
        assert np.array_equal(x[..., 40:40 + n], y)


def test_trial_group_does_not_slow_a_batch_down(sms, workloads, gpu_lib):
    """Every accepted trial group leaves the batch at its default speed (8 lanes
    a warp took 1.8 times as long) and its results as they are."""
    import torch
    W = workloads
    n = 200000
    q = torch.from_numpy(W.water_queries(n)).cuda()
    v = torch.zeros(3, n, device="cuda")
    c, w = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    ctx = sms.Context(sms.Scene(W.water_scene(res=128)), W.water_config())
    ss = sms.SpecularManifoldSingleScatter(ctx)
    ctx.set_profiling(True)

    def best(group):
        ctx.set_trial_group(group)
        ms = []
        for _ in range(5):
            ctx.reset_stats()
            ss.specular_manifold_sampling_device(q.data_ptr(), n, v.data_ptr(), c.data_ptr(), w.data_ptr(), seed=2)
            ms.append(ctx.profile()["ss_trials"]["ms"])
        return min(ms), c.cpu().numpy()

    base, counts = best(0)
    for group in (8, 16, 32):
        ms, got = best(group)
        assert np.array_equal(counts, got)
        assert ms < 1.25 * base, (group, ms, base)
    ctx.close()
