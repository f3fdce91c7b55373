"""The work that a program has this library do, as cases that can be timed and compared.

A case names one kind of call and its sizes.  The kinds, and what each stands for in use:

* ``query``    - visibility and closest-hit queries on host arrays (picking, baking probes, a host
                 integrator that only traces on the GPU): Scene.trace, both query types.
* ``query_gpu``- the same queries on rays that live on the device (Scene.trace_device).
* ``path``     - one film through PathIntegrator.render with the image read back: the Cornell box in
                 both estimator modes, the production scene, the reference's example program, the
                 textured room; independent or stratified sampler, pinhole or thin lens.
* ``tree``     - one film through WhittedIntegrator or DirectLightingIntegrator.
* ``guided``   - one film through render_guided with a network that a program has trained and keeps
                 frozen.
* ``network``  - the guiding network by itself: forward pass, gradient of one batch, and an epoch of
                 Adam steps over a pool of samples.
* ``batch``    - several uneven scenes through one render_batch.

Geometry is an asset: it follows from the case alone.  Cameras, sampler seeds, rays, weights and
training samples follow from the seed.  Every state builds its own scene; one context serves them
all, as in a program that renders many scenes.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from bonsai_gb300 import _abi as A
from bonsai_gb300 import gpu as G
from bonsai_gb300 import scenes as S

_CTX: list = []


def _ctx() -> G.Context:
    if not _CTX:
        _CTX.append(G.Context(0))
    return _CTX[0]


# ---------------------------------------------------------------- cases
def listed() -> list:
    return [
        # the smallest call: a thousand picking / probe rays against a small scene
        dict(name="probe_rays", kind="query", tris=20000, rays=1021),
        # the ray / BVH microbenchmark's scene and ray set, resident on the device
        dict(name="soup_rays", kind="query_gpu", tris=2097152, rays=16777216),
        # an interactive preview: one sample per pixel of a thumbnail, where launches count
        dict(name="preview", kind="path", scene="cornell", width=67, height=49, spp=1, depth=5, mode="pbrt"),
        # the Cornell box as configured
        dict(name="cornell_256", kind="path", scene="cornell", width=256, height=256, spp=16, depth=5, mode="pbrt"),
        # the same film in the reference's own estimator, over the reference's BVH
        dict(name="cornell_ref", kind="path", scene="cornell", width=256, height=256, spp=16, depth=5, mode="ref"),
        # the production scene: 1.31M triangles, 2000 spheres, four lights, depth 8
        dict(name="production_1080p", kind="path", scene="production", width=1920, height=1080, spp=16, depth=8,
             mode="pbrt"),
        # the reference's example program: UV-textured sphere under an environment map, 4 x 4 strata
        dict(name="example_1024", kind="path", scene="example", width=1024, height=1024, spp=16, depth=5, mode="pbrt"),
        # image textures, vertex normals, Oren-Nayar and plastic, thin lens, a ragged film
        dict(name="textured_room", kind="path", scene="textured", width=501, height=333, spp=9, depth=6, mode="pbrt"),
        # direct lighting on the production scene at a reduced film, ray trees behind glass
        dict(name="direct_production", kind="tree", integrator="direct", ico_level=4, width=640, height=360, spp=4,
             depth=8),
        # the slit room with a trained network: inference and guided shading at every vertex
        dict(name="guided_slit", kind="guided", width=640, height=360, spp=8, depth=10),
        # the network's own forward, backward and optimiser over one render pass's pool
        dict(name="guide_network", kind="network", queries=65536, samples=262144, batch=16384),
        # two dozen small scenes of uneven size in one call
        dict(name="batch_uneven", kind="batch", scenes=24, max_tris=40000, film=128, max_spp=16),
    ]


def _between(rng, lo: float, hi: float) -> int:
    """An integer of [lo, hi], spread over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["query", "query_gpu", "path", "path", "path", "path", "tree", "guided", "network", "batch"])
    if kind == "query":
        return dict(kind=kind, tris=_between(rng, 500, 200000), rays=_between(rng, 1, 300000))
    if kind == "query_gpu":
        return dict(kind=kind, tris=_between(rng, 10000, 1000000), rays=_between(rng, 100000, 12000000))
    if kind == "path":
        scene = rng.choice(["cornell", "cornell", "production", "example", "textured"])
        w = _between(rng, 33, 900)
        h = max(17, int(w * rng.uniform(0.5, 1.2)))
        spp = rng.choice([4, 9, 16]) if scene in ("example", "textured") else _between(rng, 1, 16)
        mode = "ref" if scene == "cornell" and rng.random() < 0.3 else "pbrt"
        return dict(kind=kind, scene=scene, width=w, height=h, spp=spp, depth=rng.randint(2, 8), mode=mode)
    if kind == "tree":
        w = _between(rng, 64, 600)
        return dict(kind=kind, integrator=rng.choice(["whitted", "direct"]), ico_level=rng.randint(2, 4), width=w,
                    height=max(33, int(w * rng.uniform(0.5, 1.0))), spp=rng.randint(1, 4), depth=rng.randint(2, 8))
    if kind == "guided":
        w = _between(rng, 96, 700)
        return dict(kind=kind, width=w, height=max(54, int(w * rng.uniform(0.5, 0.7))), spp=rng.randint(1, 8),
                    depth=rng.randint(4, 10))
    if kind == "network":
        return dict(kind=kind, queries=_between(rng, 1, 100000), samples=_between(rng, 128, 262144),
                    batch=128 * _between(rng, 16, 128))
    return dict(kind=kind, scenes=rng.randint(2, 24), max_tris=_between(rng, 2000, 40000), film=_between(rng, 32, 128),
                max_spp=_between(rng, 4, 16))


# ---------------------------------------------------------------- scenes (assets)
@functools.lru_cache(maxsize=4)
def _soup(tris: int) -> S.SceneData:
    return S.ray_soup(tris, 1)[0]


@functools.lru_cache(maxsize=4)
def _production(level: int) -> S.SceneData:
    return S.production(64, 36, 1, 8, ico_level=level)


@functools.lru_cache(maxsize=2)
def _slit() -> S.SceneData:
    return S.slit_room(64, 36, 1, 10, ico_level=4)


@functools.lru_cache(maxsize=2)
def _example() -> S.SceneData:
    return S.env_sphere(64, 64, env_w=512, env_h=256)


@functools.lru_cache(maxsize=2)
def _uneven(n: int, max_tris: int) -> list:
    return S.uneven_batch(n, seed=5, max_tris=max_tris, min_tris=1000)


def _scene_data(name: str) -> S.SceneData:
    if name == "cornell":
        return S.cornell(64, 64)
    if name == "production":
        return _production(5)
    if name == "example":
        return _example()
    return S.textured_room(64, 64)


def _camera(base: S.Camera, width: int, height: int, rng: np.random.Generator, lens: bool = False) -> S.Camera:
    """The scene's camera moved a little, as by a walk through the scene."""
    p = tuple(float(x) for x in np.asarray(base.position) + rng.uniform(-0.05, 0.05, 3))
    dist = float(np.linalg.norm(np.asarray(base.position) - np.asarray(base.look_at)))
    return S.Camera(p, base.look_at, base.up, base.fov_deg, width, height, base.near_plane, base.far_plane,
                    0.02 if lens else 0.0, dist if lens else base.focal_distance)


# ---------------------------------------------------------------- network inputs
_LAYER_OUT = (64, 64, 64, 64, 82)


def _weights(rng: np.random.Generator) -> np.ndarray:
    """Weights of a trained network's magnitude in the library's layout (biases in the column after
    the inputs, zero padding)."""
    p = np.zeros(A.BG_GUIDE_PARAMS, np.float32)
    for l, out in enumerate(_LAYER_OUT):
        fan = 78 if l == 0 else 64
        bound = math.sqrt(6.0 / fan) * (0.1 if l == 4 else 1.0)
        w = p[5120 * l:5120 * l + 80 * (64 if l < 4 else 96)].reshape(-1, 80)
        w[:out, :fan] = rng.uniform(-bound, bound, (out, fan))
        w[:out, fan] = rng.uniform(-0.1, 0.1, out)
    return p


def _unit(rng: np.random.Generator, n: int) -> np.ndarray:
    v = rng.normal(size=(n, 3))
    return (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(np.float32)


def _samples(rng: np.random.Generator, n: int) -> np.ndarray:
    """Training samples as a render records them: query, direction, BSDF pdf, heavy-tailed weights of
    both heads, many of them zero."""
    s = np.zeros((n, 16), np.float32)
    s[:, 0:3] = rng.random((n, 3), dtype=np.float32)
    s[:, 3:6], s[:, 6:9], s[:, 9:12] = _unit(rng, n), _unit(rng, n), _unit(rng, n)
    s[:, 12] = rng.exponential(0.3, n)
    s[:, 13] = np.where(rng.random(n) < 0.2, 0.0, rng.lognormal(0.0, 1.0, n))
    s[:, 14] = np.where(rng.random(n) < 0.6, 0.0, rng.lognormal(0.5, 1.5, n))
    return s


# ---------------------------------------------------------------- prepare / run
def _rays_gpu(n: int, seed: int) -> torch.Tensor:
    """(n, 8) bg_ray records on the device: origins uniform on the unit cube's surface, directions
    uniform on the sphere, t_max infinite."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    org = torch.rand(n, 3, generator=g, device="cuda")
    axis = torch.randint(0, 3, (n, 1), generator=g, device="cuda")
    side = torch.randint(0, 2, (n, 1), generator=g, device="cuda").float()
    org.scatter_(1, axis, side)
    d = torch.randn(n, 3, generator=g, device="cuda")
    rays = torch.zeros(n, 8, device="cuda")
    rays[:, 0:3] = org
    rays[:, 3] = float("inf")
    rays[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    return rays


def prepare(case: dict, seed: int) -> dict:
    ctx, rng, kind = _ctx(), np.random.default_rng(seed), case["kind"]
    st = dict(kind=kind, ctx=ctx)
    if kind == "query":
        st["scene"] = G.Scene(ctx, _soup(case["tris"]), A.BG_BVH_WIDE)
        st["rays"] = S.random_rays(case["rays"], seed)
    elif kind == "query_gpu":
        n = case["rays"]
        st["scene"] = G.Scene(ctx, _soup(case["tris"]), A.BG_BVH_WIDE)
        st["rays"] = _rays_gpu(n, seed)
        st["hits"] = torch.zeros(n, 2, dtype=torch.int32, device="cuda")
        st["occ"] = torch.zeros(n, dtype=torch.uint8, device="cuda")
    elif kind == "path":
        sd = _scene_data(case["scene"])
        ref = case["mode"] == "ref"
        cam = _camera(sd.camera, case["width"], case["height"], rng, lens=case["scene"] == "textured")
        sampler = None
        if case["scene"] == "example":
            side = math.isqrt(case["spp"])
            sampler = S.StratifiedSampler(side, side, 4, True)
        st["scene"] = G.Scene(ctx, sd, A.BG_BVH_REFERENCE if ref else A.BG_BVH_WIDE)
        st["integrator"] = G.PathIntegrator(cam, case["spp"], case["depth"], sd.rr_threshold, seed=seed,
                                            mode=A.BG_MODE_REF_COMPAT if ref else A.BG_MODE_PBRT, sampler=sampler)
    elif kind == "tree":
        sd = _production(case["ico_level"])
        cam = _camera(sd.camera, case["width"], case["height"], rng)
        cls = G.WhittedIntegrator if case["integrator"] == "whitted" else G.DirectLightingIntegrator
        st["scene"] = G.Scene(ctx, sd, A.BG_BVH_WIDE)
        st["integrator"] = cls(cam, case["spp"], case["depth"], seed=seed)
    elif kind == "guided":
        sd = _slit()
        cam = _camera(sd.camera, case["width"], case["height"], rng)
        st["scene"] = G.Scene(ctx, sd, A.BG_BVH_WIDE)
        st["guide"] = G.Guide(ctx, warmup_passes=0, no_train=True, no_fallback=True)
        st["guide"].params = _weights(rng)
        st["integrator"] = G.PathIntegrator(cam, case["spp"], case["depth"], sd.rr_threshold, seed=seed)
    elif kind == "network":
        st["guide"] = G.Guide(ctx, batch_size=case["batch"])
        st["weights"] = _weights(rng)
        st["queries"] = np.concatenate([rng.random((case["queries"], 3), dtype=np.float32),
                                        _unit(rng, case["queries"]), _unit(rng, case["queries"])], axis=1)
        st["samples"] = _samples(rng, case["samples"])
        st["batch"] = min(case["batch"], case["samples"])
    else:
        st["jobs"] = []
        for k, sd in enumerate(_uneven(case["scenes"], case["max_tris"])):
            w = max(8, case["film"] * (1 + k % 3) // 3)
            cam = _camera(sd.camera, w, max(8, w * (2 + k % 2) // 3), rng)
            st["jobs"].append(G.BatchJob(G.Scene(ctx, sd, A.BG_BVH_WIDE), cam, 1 + sd.spp % case["max_spp"],
                                         sd.max_depth, seed=seed + k))
    return st


def run(st: dict):
    kind = st["kind"]
    if kind == "query":
        hits = st["scene"].trace(st["rays"])
        return {"prim": hits["prim"], "t": hits["t"], "occluded": st["scene"].trace(st["rays"], any_hit=True)}
    if kind == "query_gpu":
        n, rays = st["rays"].shape[0], st["rays"].data_ptr()
        st["scene"].trace_device(rays, n, st["hits"].data_ptr())
        st["scene"].trace_device(rays, n, st["occ"].data_ptr(), any_hit=True)
        return {"prim": st["hits"][:, 0], "t": st["hits"].view(torch.float32)[:, 1], "occluded": st["occ"]}
    if kind in ("path", "tree"):
        return st["integrator"].render(st["scene"]).rgb
    if kind == "guided":
        return st["integrator"].render_guided(st["scene"], st["guide"]).rgb
    if kind == "network":
        g = st["guide"]
        g.params = st["weights"]
        out = g.forward(st["queries"])
        grad, loss = g.gradient(st["samples"][:st["batch"]])
        g.train(st["samples"])
        return {"out": out, "grad": grad, "loss": loss, "params": g.params}
    return G.render_batch(st["ctx"], st["jobs"])[0]


# ---------------------------------------------------------------- what a pass cannot do without
_RAY_FLOPS = 16 * 8 * 16 + 4 * 60  # 16 eight-wide nodes of 8 slab tests, 4 primitives
_NET_FLOPS = 2 * (80 * 64 * 4 + 80 * 82)


def _scene_bytes(tris: int, spheres: int = 0) -> int:
    return 36 * tris + 16 * spheres


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("query", "query_gpu"):
        n = case["rays"]
        return {"bytes": 2 * 32 * n + 9 * n + 2 * _scene_bytes(case["tris"]), "flops": 2 * n * _RAY_FLOPS}
    if kind == "network":
        b, n, q = min(case["batch"], case["samples"]), case["samples"], case["queries"]
        return {"bytes": 36 * q + 4 * 82 * q + 64 * (b + n) + 3 * 4 * A.BG_GUIDE_PARAMS,
                "flops": q * _NET_FLOPS + 3 * (b + n) * _NET_FLOPS}
    if kind == "batch":
        px = rays = tris = 0
        for k, sd in enumerate(_uneven(case["scenes"], case["max_tris"])):
            w = max(8, case["film"] * (1 + k % 3) // 3)
            px += w * max(8, w * (2 + k % 2) // 3)
            rays += w * max(8, w * (2 + k % 2) // 3) * (1 + sd.spp % case["max_spp"]) * 4
            tris += sd.ntri
        return {"bytes": 12 * px + _scene_bytes(tris), "flops": rays * _RAY_FLOPS}
    px = case["width"] * case["height"]
    samples = px * case["spp"]
    if kind == "tree":
        tris = 64 * 20 * 4 ** case["ico_level"]
        return {"bytes": 12 * px + _scene_bytes(tris, 2000), "flops": samples * 16 * _RAY_FLOPS}
    if kind == "guided":
        tris = 10 * 20 * 4 ** 4
        return {"bytes": 12 * px + _scene_bytes(tris, 200),
                "flops": samples * case["depth"] * (2 * _RAY_FLOPS + 0.7 * _NET_FLOPS)}
    tris = {"cornell": 12, "production": 1310730, "example": 0, "textured": 332}[case["scene"]]
    # rays per sample: a camera ray, and at each vertex a shadow ray and the next one until the path
    # leaves the scene or ends
    per = {"cornell": 1.6 * min(case["depth"], 5) + 1, "production": 4.0, "example": 1.5,
           "textured": 1.6 * min(case["depth"], 6) + 1}[case["scene"]]
    flops = _RAY_FLOPS if case["scene"] == "production" else 500
    return {"bytes": 12 * px + _scene_bytes(tris, 2000), "flops": samples * per * flops}


# ---------------------------------------------------------------- 64-bit values
def _forward64(w: list, q: torch.Tensor) -> torch.Tensor:
    k = 2.0 ** torch.arange(12, dtype=torch.float64)
    ang = math.pi * q[:, 0:3, None] * k
    x = torch.stack([torch.sin(ang), torch.cos(ang)], dim=3).reshape(len(q), 72)
    x = torch.cat([x, q[:, 3:9]], dim=1)
    one = torch.ones(len(q), 1, dtype=torch.float64)
    for l in range(5):
        x = torch.cat([x, one], dim=1) @ w[l].T
        if l < 4:
            x = torch.relu(x)
    return x


def _split64(p: np.ndarray) -> list:
    t = torch.from_numpy(p.astype(np.float64))
    return [t[5120 * l:5120 * l + 80 * out].reshape(out, 80)[:, :79 if l == 0 else 65].clone().requires_grad_()
            for l, out in enumerate(_LAYER_OUT)]


def _loss64(raw: torch.Tensor, s: torch.Tensor) -> torch.Tensor:
    """The batch loss: per head the blend (1/2, 1/2) of the one-sample mixture's and the guide's
    cross entropy against the head's weights, normalised over the batch."""
    total = torch.zeros((), dtype=torch.float64)
    for h in range(2):
        r = raw[:, 41 * h:41 * h + 41]
        lobes = r[:, :40].reshape(-1, 8, 5)
        mu = lobes[:, :, :3] / lobes[:, :, :3].norm(dim=2, keepdim=True)
        lk = lobes[:, :, 3].clamp(-2.0, 8.0)
        kap = lk.exp()
        logc = lk - math.log(2 * math.pi) - torch.log(-torch.expm1(-2 * kap))
        dotw = (mu * s[:, None, 9:12]).sum(2)
        lq = torch.logsumexp(torch.log_softmax(lobes[:, :, 4], 1) + logc + kap * (dotw - 1), 1)
        c = 0.95 * torch.sigmoid(r[:, 40])
        lmix = torch.logaddexp(c.log() + lq, torch.log((1 - c) * s[:, 12]))
        w = s[:, 13 + h]
        total = total - (w / w.sum() * 0.5 * (lmix + lq)).sum()
    return total


def exact(case: dict, seed: int):
    """The network's forward pass, gradient and loss.  The renders and ray queries have no value in 64
    bits apart from the traversal's own: their paths follow from 32-bit arithmetic."""
    if case["kind"] != "network":
        return None
    rng = np.random.default_rng(seed)
    p = _weights(rng)
    q = np.concatenate([rng.random((case["queries"], 3), dtype=np.float32), _unit(rng, case["queries"]),
                        _unit(rng, case["queries"])], axis=1)
    s = torch.from_numpy(_samples(rng, case["samples"])[:min(case["batch"], case["samples"])].astype(np.float64))
    w = _split64(p)
    with torch.no_grad():
        out = _forward64(w, torch.from_numpy(q.astype(np.float64)))
    loss = _loss64(_forward64(w, s[:, :9]), s)
    loss.backward()
    grad = np.zeros(A.BG_GUIDE_PARAMS)
    for l, o in enumerate(_LAYER_OUT):
        n = 79 if l == 0 else 65
        grad[5120 * l:5120 * l + 80 * o].reshape(o, 80)[:, :n] = w[l].grad.numpy()
    return {"out": out.numpy(), "grad": grad, "loss": float(loss), "params": None}
