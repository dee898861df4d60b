"""Chains of one to four vertices give the same bits as when these digests were
taken (tests/golden/chain_digests.json: SHA-1 of values, counts and walks, from
the kernels with one warp per query and unrolled chain traces).  Walks between
wavy faces are chaotic: a last-bit difference in a kernel, for instance from
another choice of fused multiply-adds, reaches another solution for some of
these 20,011 points, and counts change.

Four of the 136 digests are newer, those of the trial stream (sms_trials.cuh) for
chains of four vertices: unbiased with half-vector constraints, smooth and
normal-mapped (19 and 14 queries differ from the older kernels' results), and
unbiased with the angle difference, rough (187; with mnee_init 70).

Run as a script on a GB300 it prints the digests of the library as built."""
import hashlib
import json
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GOLDEN = Path(__file__).resolve().parent / "golden" / "chain_digests.json"
N = 20011


def stack_scene(sms, W, bounces, res=96, alpha=0.0, normal_mapped=False):
    """`bounces` wavy faces above the receiver, dielectrics of alternating
    sides; the topmost is the caster, the others bouncers."""
    d = sms.SceneDesc()
    for i in range(bounces):
        flip = (i % 2 == 0) if bounces % 2 == 0 else (i % 2 == 1)
        P, N_, UV, F = W.heightfield_mesh(res, 1.0, 1.0 + 0.25 * i, W.slab_waves(4 + i), flip_normals=flip)
        top = i == bounces - 1
        sid = d.add_mesh(P, F, sms.Bsdf(sms.BSDF_DIELECTRIC, 1.4, alpha=alpha),
                         sms.SHAPE_CAUSTIC_CASTER_MULTI if top else sms.SHAPE_CAUSTIC_BOUNCER, N=N_, UV=UV)
        if normal_mapped and top:
            d.normalmap = (sid, W.nm_plane_slopes(64, amp=0.02), 1.0)
    d.add_point_emitter((0.0, 0.0, 5.0), (100.0,) * 3, sms.EMITTER_CAUSTIC_MULTI)
    return d


def receiver_scene(sms, W, bounces, normal_mapped):
    """stack_scene over a diffuse floor, lit by a sphere as well."""
    d = stack_scene(sms, W, bounces, res=48, normal_mapped=normal_mapped)
    P = np.array([[-2, -2, 0], [2, -2, 0], [2, 2, 0], [-2, 2, 0]], np.float32)
    uv = np.array([[0, 0], [1, 0], [1, 1], [0, 1]], np.float32)
    d.add_mesh(P, np.array([[0, 1, 2], [0, 2, 3]], np.uint32), sms.Bsdf(sms.BSDF_DIFFUSE, 1.0, 0.0, (0.5,) * 3),
               sms.SHAPE_CAUSTIC_RECEIVER, UV=uv)
    light = d.add_sphere((0.0, 0.0, 5.0), 0.4, sms.Bsdf(sms.BSDF_DIFFUSE, 1.0, 0.0, (0.0,) * 3), 0)
    d.add_area_emitter(light, (40.0,) * 3, sms.EMITTER_CAUSTIC_MULTI)
    return d


def _sha(*arrays):
    h = hashlib.sha1()
    for a in arrays:
        h.update(np.ascontiguousarray(a).tobytes())
    return h.hexdigest()


def digests(sms, W, bounces, surface):
    """{call: digest} of one scene: connections, walks, and an image whose
    emitter hits take the unbiased-MNEE test."""
    out = {}
    scene = sms.Scene(stack_scene(sms, W, bounces, alpha=0.05 if surface == "rough" else 0.0,
                                  normal_mapped=surface == "normalmap"))
    q = W.slab_queries(N)
    for halfvector in (False, True):
        for mnee in (False, True):
            opts = dict(bounces=bounces, max_iterations=30, halfvector_constraints=halfvector, mnee_init=mnee)
            tag = f"halfvector={int(halfvector)} mnee={int(mnee)}"
            for biased in (True, False):
                ctx = sms.Context(scene, sms.SMSConfig(biased=biased, max_trials=32 if biased else 64, **opts))
                r = sms.SpecularManifoldMultiScatter(ctx).specular_manifold_sampling(q, seed=5)
                out[f"{'biased' if biased else 'unbiased'} {tag}"] = _sha(*r)
                ctx.close()
            if surface != "rough":
                ctx = sms.Context(scene, sms.SMSConfig(**opts))
                n = 8192
                w = np.zeros((8, n), np.float32)
                w[2] = 5.0
                w[6], w[7] = W.pcg32_streams_f32(11, np.arange(n, dtype=np.uint64), 2)
                out[f"walks {tag}"] = _sha(sms.SpecularManifoldMultiScatter(ctx).sample_path(
                    bounces - 1, W.slab_queries(n), w))
                ctx.close()
    if surface != "rough":
        ctx = sms.Context(sms.Scene(receiver_scene(sms, W, bounces, surface == "normalmap")),
                          sms.SMSConfig(max_trials=16, bounces=bounces, mnee_init=True))
        cam = sms.Camera.look_at((0.0, -1.2, 0.6), (0.0, 0.0, 0.1), (0.0, 0.0, 1.0), 60.0, 300, 200)
        out["image"] = _sha(ctx.render(cam, sms.RenderOptions(integrator="path_sms_ms", spp=4, seed=9, max_depth=12)))
        ctx.close()
    return out


CASES = [(b, s) for b in (1, 2, 3, 4) for s in ("smooth", "rough", "normalmap")]


@pytest.mark.parametrize("bounces, surface", CASES)
def test_same_bits(sms, workloads, gpu_lib, bounces, surface):
    want = json.loads(GOLDEN.read_text())[f"{bounces} {surface}"]
    got = digests(sms, workloads, bounces, surface)
    assert got == want, sorted(k for k in want if got.get(k) != want[k])


if __name__ == "__main__":
    import sys
    sys.path.insert(0, str(Path(__file__).resolve().parent))
    from conftest import load_package
    pkg = load_package()
    from sms_gb300 import workloads
    print(json.dumps({f"{b} {s}": digests(pkg, workloads, b, s) for b, s in CASES}, indent=1))
