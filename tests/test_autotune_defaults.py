"""The autotuners keep the library's own launch shape (blocks per SM 0) where it
is the fastest: on a context whose profile says so (no device needed)."""
import pytest


class _Context:
    """Profiles `default_ms` at the library's own blocks per SM, 1 ms elsewhere."""

    def __init__(self, default_ms):
        self.default_ms, self.blocks = default_ms, 0

    def set_launch(self, blocks, threads):
        self.blocks = blocks

    def profile(self):
        ms = self.default_ms if self.blocks == 0 else 1.0
        return {p: {"ms": ms} for p in ("ss_first", "ss_trials", "ms", "glints")}

    def set_profiling(self, on):
        pass

    def reset_stats(self):
        pass

    set_trial_group = set_treelet = set_queue_chunk = set_profiling


class _Estimator:
    def __init__(self, ctx):
        pass

    def specular_manifold_sampling_device(self, *args, seed):
        pass


@pytest.mark.parametrize("kind", ["ss", "ms", "glints"])
@pytest.mark.parametrize("default_ms, keeps", [(0.5, True), (2.0, False)])
def test_default_blocks_are_a_candidate(sms, kind, default_ms, keeps):
    from sms_gb300.autotune import autotune_blocks, autotune_ss
    module = type("Module", (), {n: _Estimator for n in ("SpecularManifoldSingleScatter",
                                                         "SpecularManifoldMultiScatter", "SpecularManifoldGlints")})
    ctx = _Context(default_ms)
    if kind == "ss":
        best = autotune_ss(module, ctx, 0, 1, 0, 0, 0)["best"][0]
    else:
        best = autotune_blocks(module, ctx, kind, 0, 1, 0, 0, 0)["best"]
    assert best == ctx.blocks and (best == 0) == keeps
