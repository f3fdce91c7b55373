"""Traversal where its shortcuts could go wrong.

Spheres: the wide layouts test them without interval arithmetic where that decides nothing, the
reference layout with it; both must give the same bits (the distance is the same sequence of
operations, and a decision is only taken early when the intervals could not change it).  The rays
start on, inside and just off a sphere, graze it, or end (t_max) at its distance and one ulp before.

Boxes: axis-aligned flat geometry at several scales, rays with zero direction components: every
plane of the node test is degenerate somewhere.  Expected hits are analytic.
"""
import numpy as np
import pytest

from bonsai_gb300 import _abi as A
from bonsai_gb300 import gpu as G
from bonsai_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def _scene(tri, spheres) -> S.SceneData:
    n = len(tri)
    return S.SceneData(np.asarray(tri, np.float32).reshape(n, 9), np.zeros(n, np.uint32), np.full(n, -1, np.int32),
                       spheres, np.stack([S.material(S.MATTE, kd=(0.5, 0.5, 0.5))]), np.zeros(0, S.LIGHT_DT))


def _rays(org, d, tmax=np.inf) -> np.ndarray:
    r = np.zeros(len(org), S.RAY_DT)
    r["org"], r["dir"], r["tmax"] = org, d, tmax
    return r


# (radius 1e-3 at 1000 is left out: there a sphere's error bound on the ray's origin is a third of its
# radius, and hits outside the sphere's box depend on each layout's boxes)
@pytest.mark.parametrize("radius,offset", [(1e-3, 0.0), (1e-3, 3.0), (0.25, 0.0), (0.25, 3.0), (0.25, 1000.0),
                                           (400.0, 0.0), (400.0, 3.0), (400.0, 1000.0)])
def test_spheres_without_intervals_equal_the_interval_test(gpu_ctx, radius, offset):
    rng = np.random.default_rng(11)
    g = np.stack(np.meshgrid(*[np.arange(3)] * 3), -1).reshape(-1, 3) * (4.0 * radius) + offset
    sph = np.zeros(len(g), S.SPHERE_DT)
    sph["center"], sph["radius"], sph["light_id"] = g, radius, -1
    sd = _scene(np.zeros((0, 9)), sph)
    n = 40_000
    d = rng.standard_normal((n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    out = rng.standard_normal((n, 3))
    out /= np.linalg.norm(out, axis=1, keepdims=True)
    c = g[rng.integers(0, len(g), n)]
    k = np.arange(n) % 4
    # on the surface, at the centre, beside the surface by up to 1e-5 radii, anywhere in the grid
    scale = np.choose(k, [1.0, 0.0, 1.0 + 1e-5 * rng.uniform(-1, 1, n), 1.0])[:, None]
    org = np.where((k == 3)[:, None], rng.uniform(offset - 4 * radius, offset + 12 * radius, (n, 3)), c + radius * scale * out)
    # every eighth ray grazes: perpendicular to the surface normal, from afar
    graze = np.arange(n) % 8 == 0
    tang = np.cross(out, d)
    tang /= np.linalg.norm(tang, axis=1, keepdims=True)
    d = np.where(graze[:, None], tang, d)
    org = np.where(graze[:, None], c + radius * (1.0 + 1e-6 * rng.uniform(-1, 1, n))[:, None] * out - 3 * radius * tang, org)
    rays = _rays(org.astype(np.float32), d.astype(np.float32))
    ref, wide, wide2 = (G.Scene(gpu_ctx, sd, b) for b in (A.BG_BVH_REFERENCE_FIXED, A.BG_BVH_WIDE, A.BG_BVH_WIDE2))
    hits = ref.trace(rays)
    assert 0.2 < (hits["prim"] >= 0).mean() < 1.0
    for tmax in (np.full(n, np.inf, np.float32), hits["t"], np.nextafter(hits["t"], np.float32(0.0))):
        rays["tmax"] = tmax
        want, occ = ref.trace(rays), ref.trace(rays, any_hit=True)
        for sc in (wide, wide2):
            got = sc.trace(rays)
            assert np.array_equal(got["prim"], want["prim"]) and np.array_equal(got["t"], want["t"])
            assert np.array_equal(sc.trace(rays, any_hit=True), occ)


@pytest.mark.parametrize("scale", [1e-4, 1.0, 1e7])
def test_flat_boxes_and_axis_rays(gpu_ctx, scale):
    # 40 parallel quads z = 1 .. 40 (two triangles each) of growing width, in units of `scale`
    tri = []
    for z in range(1, 41):
        w = 0.5 + 0.25 * z
        a, b, c, e = (-w, -w, z), (w, -w, z), (w, w, z), (-w, w, z)
        tri += [(*a, *b, *c), (*a, *c, *e)]
    sd = _scene(np.asarray(tri) * scale, np.zeros(0, S.SPHERE_DT))
    rng = np.random.default_rng(3)
    n = 4096
    # off the quads' edges and diagonals, x and y multiples of 1/8 plus 1/16, shifted apart
    x = (rng.integers(-80, 80, n) / 8.0 + 1 / 16.0)
    y = (rng.integers(-80, 80, n) / 8.0 + 1 / 32.0)
    up = rng.integers(0, 2, n) == 0
    z0 = np.where(up, 0.0, 41.0)
    org = np.stack([x, y, z0], 1) * scale
    d = np.zeros((n, 3))
    d[:, 2] = np.where(up, 1.0, -1.0)
    reach = np.maximum(np.abs(x), np.abs(y))
    first = np.clip(np.ceil((reach - 0.5) / 0.25), 1, None)  # the lowest quad that spans (x, y)
    hit = first <= 40
    want = np.where(up, first, 41.0 - 40.0)
    rays = _rays(org.astype(np.float32), d.astype(np.float32))
    for bvh in (A.BG_BVH_WIDE, A.BG_BVH_WIDE2):
        sc = G.Scene(gpu_ctx, sd, bvh)
        got = sc.trace(rays)
        assert np.array_equal(got["prim"] >= 0, hit)
        assert np.allclose(got["t"][hit], (want * scale)[hit], rtol=1e-5)
        assert np.array_equal(got["prim"][hit] // 2, np.where(up, first - 1, 39)[hit])
        assert np.array_equal(sc.trace(rays, any_hit=True) != 0, hit)


@pytest.mark.parametrize("n", [1, 2, 31, 33, 4863, 4864, 4865, 9729, 155647, 155649])
def test_short_ray_queues(gpu_ctx, n):
    """Ray counts around one ray per warp of the persistent grid, two, and full warps: every ray gets the
    hit it gets in a long queue (the same walk, so the same bits)."""
    sd, rays = S.ray_soup(3000, 160_000)
    for bvh in (A.BG_BVH_WIDE, A.BG_BVH_WIDE2):
        sc = G.Scene(gpu_ctx, sd, bvh)
        full, occ = sc.trace(rays), sc.trace(rays, any_hit=True)
        got = sc.trace(rays[:n])
        assert np.array_equal(got["prim"], full["prim"][:n]) and np.array_equal(got["t"], full["t"][:n])
        assert np.array_equal(sc.trace(rays[:n], any_hit=True), occ[:n])
