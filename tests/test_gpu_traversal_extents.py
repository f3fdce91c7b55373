"""The 8-wide layout's node test in very large scenes: a zero direction component (an inverse of 1e20)
times a node's extent comes near the end of FP32.  Spheres (whose own test still has range there) hit by
rays along an axis and within a coordinate plane; the reference layout, whose slabs divide by the
component itself, says what is hit."""
import numpy as np
import pytest

from bonsai_gb300 import _abi as A
from bonsai_gb300 import gpu as G
from bonsai_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log2_extent", [0, 40, 58, 59, 60, 61])
def test_axis_rays_at_large_extents(gpu_ctx, log2_extent):
    ext, n, m = 2.0 ** log2_extent, 64, 4096
    rng = np.random.default_rng(1)
    centre = rng.random((n, 3)) * ext
    centre[0], centre[1] = 0.0, ext
    sph = np.zeros(n, S.SPHERE_DT)
    sph["center"], sph["radius"], sph["light_id"] = centre, ext / 20, -1
    sd = S.SceneData(np.zeros((0, 9), np.float32), np.zeros(0, np.uint32), np.zeros(0, np.int32), sph,
                     np.stack([S.material(S.MATTE, kd=(0.5, 0.5, 0.5))]), np.zeros(0, S.LIGHT_DT))
    axis = rng.integers(0, 3, m)
    d = np.zeros((m, 3))
    d[np.arange(m), axis] = rng.choice([-1.0, 1.0], m)
    slanted = np.arange(m) % 2 == 0  # half of the rays lie in a coordinate plane instead
    d[slanted, axis[slanted]] *= 0.8
    d[slanted, (axis[slanted] + 1) % 3] = rng.choice([-0.6, 0.6], int(slanted.sum()))
    rays = np.zeros(m, S.RAY_DT)
    rays["org"], rays["dir"], rays["tmax"] = rng.random((m, 3)) * ext, d, np.inf
    ref = G.Scene(gpu_ctx, sd, A.BG_BVH_REFERENCE_FIXED)
    want, occ = ref.trace(rays), ref.trace(rays, any_hit=True)
    assert (want["prim"] >= 0).sum() > 500
    sc = G.Scene(gpu_ctx, sd, A.BG_BVH_WIDE)
    got = sc.trace(rays)
    assert np.array_equal(got["prim"], want["prim"]) and np.array_equal(got["t"], want["t"])
    assert np.array_equal(sc.trace(rays, any_hit=True), occ)
