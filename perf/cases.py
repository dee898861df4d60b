"""Workloads of the SMS library, each one call (or one short call sequence) of its public Python
entry points: caustic connections over device and host query batches, two-bounce chains, glints,
normal-mapped casters, whole images, and one training gradient of the learned seed proposal.

Scenes are those of specular-manifold-sampling_gb300/workloads.py.  A program builds a scene and
its context once and then sends query batches to it, so contexts are kept between preparations;
queries, sampler seeds, images and buffers are new for every seed."""
import functools
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

PKG = Path(__file__).resolve().parents[1] / "specular-manifold-sampling_gb300"


def _package():
    """The package directory's name is no identifier: import it as sms_gb300."""
    if "sms_gb300" not in sys.modules:
        spec = importlib.util.spec_from_file_location("sms_gb300", PKG / "__init__.py",
                                                      submodule_search_locations=[str(PKG)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["sms_gb300"] = mod
        spec.loader.exec_module(mod)
    from sms_gb300 import workloads
    return sys.modules["sms_gb300"], workloads


def listed():
    return [
        # caustic of a mirror sphere on a 64 x 64 receiver grid, biased: the smallest device batch
        {"name": "sphere_grid", "kind": "sphere", "n": 4096, "trials": 16},
        # a full frame of shading points under the 512^2 water surface, unbiased (the headline workload)
        {"name": "water_frame", "kind": "water", "n": 1 << 20, "res": 512, "trials": 256, "alpha": 0.0},
        # one ragged tile of a frame, a coarser surface
        {"name": "water_tile", "kind": "water", "n": 32003, "res": 256, "trials": 256, "alpha": 0.0},
        # a renderer on the host asks for the shading points of one small block: host arrays in and out
        {"name": "water_host_block", "kind": "water_host", "n": 300, "res": 128, "trials": 256, "alpha": 0.0},
        # a rough (Beckmann) water surface: offset normals in every walk
        {"name": "water_rough", "kind": "water", "n": 16384, "res": 128, "trials": 64, "alpha": 0.1},
        # two refractions through a glass slab, biased, 32 walks a point
        {"name": "slab_biased", "kind": "slab", "n": 65536, "res": 256, "biased": True, "trials": 32, "bounces": 2},
        # the same chains by the unbiased estimator, an odd batch
        {"name": "slab_unbiased", "kind": "slab", "n": 20011, "res": 256, "biased": False, "trials": 128,
         "bounces": 2},
        # the glints of one frame on a large slope map, vectorized estimator
        {"name": "glint_frame", "kind": "glints", "width": 700, "map": 4096, "trials": 64, "biased": True},
        # a normal-mapped glass pane with the two-stage solver
        {"name": "pane_twostage", "kind": "pane", "n": 30000, "map": 256, "biased": False, "trials": 64,
         "twostage": True, "conductor": False},
        # a preview image of the pool with SMS caustics
        {"name": "render_caustics", "kind": "render", "integrator": "path_sms_ss", "res": 256, "width": 192,
         "height": 160, "spp": 8},
        # the same scene by plain path tracing, at film size
        {"name": "render_path", "kind": "render", "integrator": "path", "res": 512, "width": 512, "height": 384,
         "spp": 16},
        # loss and gradient of the seed proposal over one training batch
        {"name": "proposal_gradient", "kind": "gradient", "n": 8192},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sphere", "water", "water", "water_host", "slab", "slab", "glints", "pane", "render",
                       "gradient"])
    if kind == "sphere":
        return {"kind": kind, "n": _log(rng, 700, 60000), "trials": rng.choice([8, 16, 24, 32])}
    if kind == "water":
        return {"kind": kind, "n": _log(rng, 1000, 600000), "res": rng.choice([64, 128, 200, 256, 512]),
                "trials": rng.choice([32, 100, 256]), "alpha": rng.choice([0.0, 0.0, 0.0, 0.1])}
    if kind == "water_host":
        return {"kind": kind, "n": _log(rng, 30, 4000), "res": rng.choice([64, 128, 256]),
                "trials": rng.choice([64, 256]), "alpha": 0.0}
    if kind == "slab":
        return {"kind": kind, "n": _log(rng, 500, 50000), "res": rng.choice([64, 128, 256]),
                "biased": rng.random() < 0.5, "trials": rng.choice([8, 16, 32, 48]), "bounces": 2}
    if kind == "glints":
        return {"kind": kind, "width": _log(rng, 90, 1000), "map": rng.choice([512, 1024, 2048, 4096]),
                "trials": rng.choice([12, 16, 32, 64]), "biased": rng.random() < 0.7}
    if kind == "pane":
        two = rng.random() < 0.5
        return {"kind": kind, "n": _log(rng, 1000, 100000), "map": rng.choice([128, 256, 512]),
                "biased": rng.random() < 0.5, "trials": rng.choice([16, 32, 64]), "twostage": two,
                "conductor": rng.random() < 0.3}
    if kind == "render":
        w = _log(rng, 48, 480)
        sms = rng.random() < 0.5
        return {"kind": kind, "integrator": "path_sms_ss" if sms else "path", "res": rng.choice([64, 128, 256]),
                "width": w, "height": max(16, int(w * rng.uniform(0.5, 1.0))),
                "spp": rng.choice([1, 2, 4]) if sms else rng.choice([4, 9, 16])}
    return {"kind": kind, "n": 16 * _log(rng, 16, 3000)}


# ------------------------------------------------------------------- contexts
def _slopes(res):
    """(res, res, 2) FP16 slopes: white noise smoothed by a Gaussian of 4 texels (periodic), std 0.15."""
    g = torch.Generator(device="cuda").manual_seed(7)
    f = torch.fft.fftfreq(res, device="cuda")
    low = torch.exp(-2.0 * (math.pi * 4.0) ** 2 * (f[:, None] ** 2 + f[None, :res // 2 + 1] ** 2))
    out = []
    for _ in range(2):
        w = torch.randn(res, res, device="cuda", generator=g)
        w = torch.fft.irfft2(torch.fft.rfft2(w) * low, s=(res, res))
        out.append((w * (0.15 / w.std())).half())
    return torch.stack(out, dim=-1).cpu().numpy()


@functools.lru_cache(maxsize=6)
def _desc(kind, a, b):
    sms, W = _package()
    if kind == "sphere":
        return W.sphere_scene(conductor=True)
    if kind == "water":
        d = W.water_scene(res=a)
        if b > 0.0:
            P, N, UV, F, bsdf, flags = d.meshes[0]
            d.meshes[0] = (P, N, UV, F, sms.Bsdf(bsdf.type, bsdf.eta, alpha=b), flags)
        return d
    if kind == "slab":
        return W.slab_scene(res=a)
    if kind == "glints":
        return W.glint_scene(map_res=a, slopes=_slopes(a))
    if kind == "pane":
        return W.nm_plane_scene(conductor=b, res=a)
    return W.pool_scene(res=a)


@functools.lru_cache(maxsize=8)
def _context(kind, a, b, config):
    sms, _ = _package()
    return sms.Context(sms.Scene(_desc(kind, a, b)), sms.SMSConfig(**dict(config)), device=0)


def _config(case):
    k = case["kind"]
    if k == "sphere":
        c = {"biased": True, "max_trials": case["trials"]}
    elif k in ("water", "water_host"):
        c = {"max_trials": case["trials"]}
    elif k == "slab":
        c = {"biased": case["biased"], "max_trials": case["trials"], "max_iterations": 30,
             "bounces": case["bounces"]}
    elif k == "glints":
        c = {"biased": case["biased"], "max_trials": case["trials"], "max_iterations": 10,
             "glints_vectorized": case["biased"]}
    elif k == "pane":
        c = {"biased": case["biased"], "max_trials": case["trials"], "twostage": case["twostage"]}
    else:
        c = {"max_trials": 64}
    return tuple(sorted(c.items()))


def _case_context(case):
    k = case["kind"]
    scene = {"sphere": ("sphere", 0, 0), "glints": ("glints", case.get("map"), 0),
             "pane": ("pane", case.get("map"), case.get("conductor", False)),
             "slab": ("slab", case.get("res"), 0), "render": ("pool", case.get("res"), 0),
             "gradient": ("water", 128, 0.0)}.get(k, ("water", case.get("res"), case.get("alpha", 0.0)))
    return _context(*scene, _config(case))


# --------------------------------------------------------------------- inputs
def _rng(seed):
    return np.random.default_rng(1000003 * 7 + seed)


def _points(case, seed):
    """(n, 2) receiver points: the sphere's and the pane's grids jittered, uniform elsewhere."""
    r, n = _rng(seed), case["n"]
    u = r.random((n, 2), dtype=np.float32)
    if case["kind"] == "sphere":
        res = math.ceil(math.sqrt(n))
        i = np.arange(n)
        cell = np.stack([i % res, i // res], axis=1)
        return ((cell + u) / res * 4.0 - 2.0).astype(np.float32)
    return ((2.0 * u - 1.0) * (0.8 if case["kind"] == "pane" else 1.0)).astype(np.float32)


def _features(case, seed):
    """Training pairs as the solver collects them: shading point, light sample and normal, the
    solution's uv near the straight path, contribution shares in (0, 1]."""
    r, n = _rng(seed), case["n"]
    xy = 2.0 * r.random((2, n)) - 1.0
    z = 1.0 - 2.0 * r.random(n)
    ph = 2.0 * np.pi * r.random(n)
    s = np.sqrt(1.0 - z * z)
    light = np.stack([0.1 * s * np.cos(ph), 0.1 * s * np.sin(ph), 10.0 + 0.1 * z])
    f = np.concatenate([xy, np.zeros((1, n)), light, np.zeros((2, n)), np.ones((1, n))]).astype(np.float32)
    uv = (0.5 * (0.9 * xy + 0.07 * r.standard_normal((2, n))) + 0.5).astype(np.float32)
    return f, uv, (1.0 - r.random(n)).astype(np.float32)


def prepare(case, seed):
    sms, W = _package()
    ctx, k = _case_context(case), case["kind"]
    st = {"kind": k, "ctx": ctx, "seed": 17 + seed}
    if k == "render":
        st["camera"] = W.pool_camera(case["width"], case["height"])
        st["options"] = sms.RenderOptions(integrator=case["integrator"], spp=case["spp"], max_depth=6,
                                          seed=st["seed"])
        return st
    if k == "gradient":
        f, uv, w = _features(case, seed)
        p = sms.SeedProposal(ctx, 0, seed=1 + seed, capacity=case["n"])
        p.set_data(f, uv, w)
        p.normalize()
        st["proposal"], st["batch"] = p, case["n"]
        return st
    if k == "glints":
        q = W.glint_queries(case["width"])
        shift = (0.02 * _rng(seed).random(2) - 0.01).astype(np.float32)
        for row in (0, 12, 18):   # the camera and what it sees move over the plane together
            q[row:row + 2] += shift[:, None]
    else:
        q = W.plane_queries(_points(case, seed))
    if k == "water_host":
        st["solver"], st["queries"] = sms.SpecularManifoldSingleScatter(ctx), q
        return st
    solver = {"slab": sms.SpecularManifoldMultiScatter, "glints": sms.SpecularManifoldGlints}
    st["solver"] = solver.get(k, sms.SpecularManifoldSingleScatter)(ctx)
    n = q.shape[1]
    st["queries"] = torch.from_numpy(q).cuda()
    st["value"] = torch.zeros(3, n, device="cuda")
    st["count"] = torch.zeros(n, dtype=torch.int32, device="cuda")
    st["walks"] = torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()   # the solver works on its context's own stream
    return st


def run(state):
    k = state["kind"]
    if k == "render":
        return state["ctx"].render(state["camera"], state["options"])
    if k == "gradient":
        loss, grad = state["proposal"].loss_grad(state["batch"])
        return [loss, grad]
    if k == "water_host":
        return list(state["solver"].specular_manifold_sampling(state["queries"], seed=state["seed"]))
    v, c, w = state["value"], state["count"], state["walks"]
    state["solver"].specular_manifold_sampling_device(state["queries"].data_ptr(), c.numel(), v.data_ptr(),
                                                      c.data_ptr(), w.data_ptr(), seed=state["seed"])
    return [v, c, w]


def work(case):
    """Bytes: queries read and results written once, and the scene (or the touched part of the slope
    map) read once.  Floating-point operations: those of the Newton iterations and the ray casts of
    the walks the estimator has to make, from the operation counts of the scalar code
    (profiles/flops_per_unit.json): about 1000 a ray on meshes, 480 on a sphere, 110 a glint step."""
    k = case["kind"]
    if k == "render":
        px = case["width"] * case["height"]
        paths = px * case["spp"]
        rays = paths * (8 + (5 * 21 if case["integrator"] == "path_sms_ss" else 0))
        return {"bytes": 12 * px + 80 * case["res"] ** 2, "flops": 1000.0 * rays}
    if k == "gradient":
        return {"bytes": 48 * case["n"] + 8 * 21808, "flops": 6.0 * 21808 * case["n"]}
    if k == "glints":
        n = 0.6 * case["width"] ** 2
        walks = case["trials"] if case["biased"] else 0.5 * case["trials"]
        return {"bytes": n * (84 + 20) + 4 * case["map"] ** 2, "flops": 110.0 * 6 * n * walks}
    n = case["n"]
    if k == "sphere":
        return {"bytes": 84.0 * n, "flops": 480.0 * 6 * n * case["trials"]}
    if k == "pane":
        walks = case["trials"] if case["biased"] else 4
        return {"bytes": 84.0 * n + 4 * case["map"] ** 2, "flops": 700.0 * 8 * n * walks}
    scene = 80.0 * case["res"] ** 2
    if k == "slab":
        walks = case["trials"] if case["biased"] else 12
        return {"bytes": 84.0 * n + 2 * scene, "flops": 2000.0 * 12 * n * walks}
    return {"bytes": 84.0 * n + scene, "flops": 1000.0 * 21 * 5 * n}


# ---------------------------------------------------------------------- exact
_M64 = np.uint64(6364136223846793005)


def _pcg_uniforms(seed, n, count):
    """count float32 uniforms of each of n PCG32 (XSH-RR 64/32) streams, as float64: (count, n)."""
    with np.errstate(over="ignore"):
        inc = (np.arange(n, dtype=np.uint64) << np.uint64(1)) | np.uint64(1)

        def step(s):
            xs = (((s >> np.uint64(18)) ^ s) >> np.uint64(27)).astype(np.uint32)
            rot = (s >> np.uint64(59)).astype(np.uint32)
            return s * _M64 + inc, (xs >> rot) | (xs << ((np.uint32(32) - rot) & np.uint32(31)))

        s, _ = step(np.zeros(n, np.uint64))
        s, _ = step(s + np.uint64(seed))
        out = np.empty((count, n))
        for i in range(count):
            s, u = step(s)
            out[i] = ((u >> np.uint32(9)) | np.uint32(0x3F800000)).view(np.float32).astype(np.float64) - 1.0
    return out


def _dot(a, b):
    return (a * b).sum(-1)


def _unit(a):
    return a / np.sqrt(_dot(a, a))[..., None]


SPHERE_C, SPHERE_LIGHT = np.array([0.0, 0.0, 1.5]), np.array([0.0, 0.0, 5.0])


def _sphere_ray(x, d):
    """Nearest hit of rays from x (outside) with the unit sphere: (hit, point)."""
    oc = x - SPHERE_C
    b = _dot(oc, d)
    disc = b * b - (_dot(oc, oc) - 1.0)
    t = -b - np.sqrt(np.maximum(disc, 0.0))
    hit = (disc >= 0.0) & (t > 0.0)
    return hit, np.where(hit[..., None], x + d * t[..., None], 0.0)


def _sphere_frame(p):
    """Normal and the tangents of the (phi, theta) parametrisation, scaled to unit uv."""
    n = p - SPHERE_C
    rd = np.maximum(np.hypot(n[..., 0], n[..., 1]), 1e-300)
    z = np.zeros_like(rd)
    du = 2 * np.pi * np.stack([-n[..., 1], n[..., 0], z], -1)
    dv = np.pi * np.stack([n[..., 2] * n[..., 0] / rd, n[..., 2] * n[..., 1] / rd, -rd], -1)
    return n, du, dv, 2 * np.pi * rd, np.pi


def _angles(w, du, dv):
    """(theta, phi) of w and their derivatives along du and dv: rows (theta, phi), columns (u, v)."""
    th, ph = np.arccos(np.clip(w[..., 2], -1, 1)), np.arctan2(w[..., 1], w[..., 0])
    ph = np.where(ph < 0, ph + 2 * np.pi, ph)
    da = -1.0 / np.sqrt(np.maximum(1.0 - w[..., 2] ** 2, 1e-300))
    q = w[..., 0] ** 2 + w[..., 1] ** 2
    dphi = [(w[..., 0] * d[..., 1] - w[..., 1] * d[..., 0]) / np.maximum(q, 1e-300) for d in (du, dv)]
    return th, ph, (da * du[..., 2], da * dv[..., 2]), dphi


def _sphere_exact(case, seed):
    """The biased estimator on the mirror sphere in float64: every walk's Newton iteration on the
    angle difference between the reflected and the light direction, the distinct solutions in walk
    order, and their contribution (Fresnel, generalised geometry term, point light, diffuse plane)."""
    n, M = case["n"], case["trials"]
    xy = _points(case, seed).astype(np.float64)
    x = np.concatenate([xy, np.zeros((n, 1))], axis=1)
    u = _pcg_uniforms(17 + seed, n, 3 + 2 * M)
    total, kept = np.zeros(n), []
    for m in range(M):
        z = 1.0 - 2.0 * u[4 + 2 * m]
        r, phi = np.sqrt(np.maximum(1.0 - z * z, 0.0)), 2 * np.pi * u[3 + 2 * m]
        goal = SPHERE_C + np.stack([r * np.cos(phi), r * np.sin(phi), z], -1)
        live, p = _sphere_ray(x, _unit(goal - x))
        beta, good, done = np.ones(n), np.zeros(n, bool), np.zeros(n, bool)
        for _ in range(20):
            nn, du, dv, _, _ = _sphere_frame(p)
            wi, wo = x - p, SPHERE_LIGHT - p
            li, lo = np.sqrt(_dot(wi, wi)), np.sqrt(_dot(wo, wo))
            wi, wo = wi / li[:, None], wo / lo[:, None]
            diff = lambda w, l, d: -(d - w * _dot(w, d)[:, None]) / l[:, None]  # noqa: E731
            iu, iv, ou, ov = diff(wi, li, du), diff(wi, li, dv), diff(wo, lo, du), diff(wo, lo, dv)
            refl = lambda dw, dn: 2 * (nn * (_dot(dw, nn) + _dot(wi, dn))[:, None]  # noqa: E731
                                       + dn * _dot(wi, nn)[:, None]) - dw
            t = nn * (2 * _dot(wi, nn))[:, None] - wi
            t0, p0, dt0, dp0 = _angles(wo, ou, ov)
            t1, p1, dt1, dp1 = _angles(t, refl(iu, du), refl(iv, dv))
            c0, c1 = t0 - t1, p0 - p1
            c1 = np.where(c1 < -np.pi, c1 + 2 * np.pi, np.where(c1 > np.pi, c1 - 2 * np.pi, c1))
            a, b, c, d = dt0[0] - dt1[0], dt0[1] - dt1[1], dp0[0] - dp1[0], dp0[1] - dp1[1]
            det = a * d - b * c
            live &= ~(np.abs(det) < 1e-6)
            conv = live & ~done & (np.hypot(c0, c1) < 1e-5)
            done |= conv
            det = np.where(det == 0, 1.0, det)
            s0, s1 = (d * c0 - b * c1) / det, (a * c1 - c * c0) / det
            step = (du * s0[:, None] + dv * s1[:, None]) * beta[:, None]
            hit, q = _sphere_ray(x, _unit(p - step - x))
            go = live & ~done
            take = go & hit
            good = np.where(go, hit, good)
            beta = np.where(take, np.minimum(1.0, 2 * beta), np.where(go, 0.5 * beta, beta))
            p = np.where(take[:, None], q, p)
        nn, du, dv, lu, lv = _sphere_frame(p)
        ok = live & done & good & (_dot(nn, x - p) * _dot(nn, SPHERE_LIGHT - p) >= 0)
        back = _unit(p - SPHERE_LIGHT)   # the light sees the solution
        h, q = _sphere_ray(np.broadcast_to(SPHERE_LIGHT, p.shape), back)
        near = np.sqrt(_dot(q - SPHERE_LIGHT, q - SPHERE_LIGHT)) < np.sqrt(_dot(p - SPHERE_LIGHT, p - SPHERE_LIGHT)) * (1 - 9e-5)
        ok &= ~(h & near)
        dirs = _unit(p - x)
        for k_ok, k_dir in kept:
            ok &= ~(k_ok & (np.abs(_dot(dirs, k_dir) - 1.0) < 1e-4))
        kept.append((ok, dirs))
        wi, wo = x - p, SPHERE_LIGHT - p
        li, lo = np.sqrt(_dot(wi, wi)), np.sqrt(_dot(wo, wo))
        wi, wo = wi / li[:, None], wo / lo[:, None]
        cos = np.abs(_dot(nn, wo))
        er, ek = float(np.float32(0.2)), float(np.float32(3.0))
        s2 = 1 - cos * cos
        k1 = er * er - ek * ek - s2
        ab = np.sqrt(np.maximum(k1 * k1 + 4 * ek * ek * er * er, 0))
        aa = np.sqrt(np.maximum(0.5 * (ab + k1), 0))
        rs = (ab + cos ** 2 - 2 * cos * aa) / (ab + cos ** 2 + 2 * cos * aa)
        rp = rs * (ab * cos ** 2 + s2 * s2 - 2 * cos * aa * s2) / (ab * cos ** 2 + s2 * s2 + 2 * cos * aa * s2)
        F = 0.5 * (rs + rp)
        # orthonormal tangents (the parametrisation is orthogonal; dn = tangent on the unit sphere)
        s, t = du / lu[:, None], dv / lv
        hv = wi + wo
        il = 1 / np.sqrt(_dot(hv, hv))
        hv, ilo, ili = hv * il[:, None], il / lo, il / li
        proj = lambda d: d - hv * _dot(d, hv)[:, None]  # noqa: E731
        dh = lambda e: proj(-e * (ili + ilo)[:, None] + wi * (_dot(wi, e) * ili)[:, None]  # noqa: E731
                            + wo * (_dot(wo, e) * ilo)[:, None])
        hn = _dot(hv, nn)
        A = [[_dot(dh(s), s) - hn, _dot(dh(t), s)], [_dot(dh(s), t), _dot(dh(t), t) - hn]]
        y = _unit(p - SPHERE_LIGHT)
        ref = np.where(np.abs(y[:, 2:3]) < 0.9, np.array([[0.0, 0.0, 1.0]]), np.array([[1.0, 0.0, 0.0]]))
        y1 = _unit(np.cross(y, ref))
        y2 = np.cross(y, y1)
        g = lambda e: proj((e - wo * _dot(wo, e)[:, None]) * ilo[:, None])  # noqa: E731
        B = [[_dot(g(y1), s), _dot(g(y2), s)], [_dot(g(y1), t), _dot(g(y2), t)]]
        dA = A[0][0] * A[1][1] - A[0][1] * A[1][0]
        dB = B[0][0] * B[1][1] - B[0][1] * B[1][0]
        ratio = np.minimum(np.abs(dB / np.where(dA == 0, 1, dA)), 1.0)
        G = np.where(np.abs(dA) < 1e-6, 0.0, np.abs(_dot(wi, nn)) / li ** 2 * ratio)
        total += np.where(ok, 100.0 * F * G * 0.5 / np.pi * np.maximum(dirs[:, 2], 0.0), 0.0)
    return [np.broadcast_to(total, (3, n)).copy(), None, None]


def _gradient_exact(case, seed):
    """Loss and gradient of the mixture network in float64 (autograd), from the parameters the
    proposal was made with; pairs, layout and anchor as the SeedProposal class documents them."""
    sms, _ = _package()
    f, uv, w = _features(case, seed)
    p = sms.SeedProposal(_case_context(case), 0, seed=1 + seed, capacity=16)
    par = torch.from_numpy(p.state()["params"]).double().cuda().requires_grad_(True)
    fr = torch.from_numpy(p.frame()).double().cuda()
    p.close()
    F, UV, Wt = (torch.from_numpy(a).double().cuda() for a in (f, uv, w))
    mean, sd = F.mean(1, keepdim=True), F.std(1, unbiased=False, keepdim=True)
    x = torch.where(sd > 1e-6 * mean.abs().clamp(min=1.0), (F - mean) / sd.clamp(min=1e-30), torch.zeros_like(F))
    cols = [x.T]
    for k in range(9):
        a = math.pi * x[k][:, None] * 2.0 ** torch.arange(4, device="cuda")
        cols += [torch.sin(a), torch.cos(a)]
    h, off = torch.cat(cols, 1), 0
    for i, o in ((96, 64), (64, 64), (64, 64), (64, 64), (64, 48)):
        Wl, b = par[off:off + o * i].reshape(o, i), par[off + o * i:off + o * i + o]
        off += o * i + o
        z = h @ Wl[:, :h.shape[1]].T + b
        h = z * torch.sigmoid(z)
    org, au, av = fr[1:4], fr[4:7], fr[7:10]
    nrm = torch.linalg.cross(au, av)
    d = F[3:6] - F[0:3]
    t = (nrm @ (org[:, None] - F[0:3])) / (nrm @ d)
    hit = F[0:3] + d * t - org[:, None]
    anchor = torch.stack([au @ hit / (au @ au), av @ hit / (av @ av)]).clamp(-1.0, 2.0)
    mu, ls = z[:, 8:24].reshape(-1, 8, 2), -7.0 + 7.0 * torch.sigmoid(z[:, 24:40].reshape(-1, 8, 2))
    e = (UV - anchor).T[:, None, :] - mu
    lp = torch.log_softmax(z[:, :8], 1) - math.log(2 * math.pi) - ls.sum(2) - 0.5 * (e * e * torch.exp(-2 * ls)).sum(2)
    loss = (-torch.logsumexp(lp, 1) * Wt).mean()
    loss.backward()
    return [float(loss), par.grad.cpu().numpy()]


def exact(case, seed):
    """Float64 results where the estimate is a well-conditioned function of its inputs.  Walks on
    wavy surfaces are chaotic (one rounding moves a walk to another solution), so connections and
    images over them have no such value."""
    if case["kind"] == "sphere":
        return _sphere_exact(case, seed) if case["n"] * case["trials"] <= 400000 else None
    if case["kind"] == "gradient":
        return _gradient_exact(case, seed)
    return None
