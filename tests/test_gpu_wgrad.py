"""Weight gradients of the learned proposal at the edges of a warp's 256 samples:
one 16-sample tile alone, whole and partial 32-sample steps, a short last chunk.
Against the oracle's bf16-emulating backward pass, with the bounds of the
gradient test in test_gpu_proposal.py (the rare bf16 rounding flips)."""
import numpy as np
import pytest

from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu
GRAD_REL, GRAD_COS = 3e-2, 0.999


@pytest.mark.parametrize("batch", [16, 32, 48, 240, 272, 528, 1040])
def test_gradient_at_chunk_edges(sms, workloads, gpu_lib, batch):
    ctx = sms.Context(sms.Scene(workloads.water_scene(res=32)), sms.SMSConfig(biased=False, max_trials=16))
    rng = np.random.default_rng(batch)
    feat = rng.normal(size=(9, batch)).astype(np.float32)
    uv = rng.uniform(0.2, 0.8, size=(2, batch)).astype(np.float32)
    p = rng.uniform(-0.2, 0.2, M.N_PARAMS).astype(np.float32)
    M.unpack(p)[0][0][:, M.N_ENC:] = 0.0
    norm = np.concatenate([rng.normal(size=9), rng.uniform(0.5, 2.0, 9)]).astype(np.float32)
    prop = sms.SeedProposal(ctx, 0, seed=3, capacity=batch)
    prop.set_data(feat, uv)
    prop.load_state({"params": p, "norm": norm, "step": 0})
    loss, grad = prop.loss_grad(batch)
    lo, go = M.loss_grad(p, norm[:9], norm[9:], feat, uv, bf=True, frame=prop.frame())
    assert abs(loss - lo) < 1e-3 * max(1.0, abs(lo))
    off = 0
    for i, o in M.LAYERS:
        for sl in (slice(off, off + o * i), slice(off + o * i, off + o * i + o)):
            g1, g2 = grad[sl].astype(np.float64), go[sl]
            rel = np.linalg.norm(g1 - g2) / max(np.linalg.norm(g2), 1e-12)
            cos = g1 @ g2 / max(np.linalg.norm(g1) * np.linalg.norm(g2), 1e-30)
            assert rel < GRAD_REL and cos > GRAD_COS, (sl, rel, cos)
        off += o * i + o
    ctx.close()
