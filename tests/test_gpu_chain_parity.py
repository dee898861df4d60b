"""Chains of one, three and four vertices against the oracle (manifold_ms.cpp):
connections by both estimators, smooth and rough faces.  Tolerances as in
test_gpu_ms_parity: count mismatches may not exceed 1.5 x the oracle-vs-FMA-oracle
floor + 0.5 %."""
import pytest

from test_gpu_chain_digests import stack_scene
from test_gpu_ss_parity import FLOOR_FACTOR, FLOOR_SLACK, _connect_diff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("biased", [True, False])
@pytest.mark.parametrize("alpha", [0.0, 0.05])
@pytest.mark.parametrize("bounces", [1, 3, 4])
def test_connections_match_the_oracle(sms, workloads, oracle, gpu_lib, bounces, alpha, biased):
    desc = stack_scene(sms, workloads, bounces, alpha=alpha)
    cfg = sms.SMSConfig(biased=biased, max_trials=16 if biased else 64, max_iterations=30, bounces=bounces)
    q = workloads.slab_queries(2048)
    ctx = sms.Context(sms.Scene(desc), cfg)
    vg, cg, wg = sms.SpecularManifoldMultiScatter(ctx).specular_manifold_sampling(q, seed=2)
    ctx.close()
    vo, co, wo, _ = oracle.OracleScene(desc).connect_batch(cfg, q, seed=2, multi=True)
    vf, cf, wf, _ = oracle.OracleScene(desc, fma=True).connect_batch(cfg, q, seed=2, multi=True)
    g_cm, g_diff, g_med = _connect_diff(vg, cg, wg, vo, co, wo)
    f_cm, f_diff, _ = _connect_diff(vf, cf, wf, vo, co, wo)
    print(f"{bounces} vertices alpha={alpha} {'biased' if biased else 'unbiased'}: count mismatch {g_cm:.4f} differs "
          f"{g_diff:.4f} (floor {f_cm:.4f}/{f_diff:.4f}) median rel {g_med:.1e}")
    assert (co > 0).any()
    assert g_cm <= FLOOR_FACTOR * f_cm + FLOOR_SLACK
    assert g_diff <= FLOOR_FACTOR * f_diff + FLOOR_SLACK
    assert g_med < 1e-4
