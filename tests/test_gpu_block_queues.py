"""Queue appends by whole blocks: wave sizes around the blocks of the binning (512 threads) and
shading (512, tree levels 1024) kernels, and around a warp.  Every path must reach the film exactly
once, whatever the remainder of the last block: a film rendered in waves of an awkward size equals
the film rendered in one wave (the same paths; the film's sums are FP64 and the resolved pixel FP32,
so an equal set of samples gives pixels equal to 1e-6 in any order of summation)."""
import numpy as np
import pytest

from bonsai_gb300 import _abi as A
from bonsai_gb300 import autotune
from bonsai_gb300 import gpu as G
from bonsai_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wave", [1024, 1025, 1535, 1537, 2047, 4099])
@pytest.mark.parametrize("kind", ["path", "textured", "whitted", "direct"])
def test_ragged_waves_equal_one_wave(gpu_ctx, kind, wave):
    sd = (S.textured_room if kind == "textured" else S.cornell)(61, 43, spp=3)
    sc = G.Scene(gpu_ctx, sd, A.BG_BVH_WIDE)
    integ = {"whitted": lambda: G.WhittedIntegrator(sd.camera, 3, 4), "direct": lambda: G.DirectLightingIntegrator(sd.camera, 3, 4)}.get(
        kind, lambda: G.PathIntegrator(sd.camera, 3, 5))()
    old = autotune.get(gpu_ctx)
    try:
        films = []
        for w in (1 << 20, wave):
            autotune.set_(gpu_ctx, old.refill, old.blocks_per_sm, w)
            films.append((integ.render(sc).rgb, G.PathIntegrator.moments(gpu_ctx, 61, 43)))
    finally:
        autotune.set_(gpu_ctx, old.refill, old.blocks_per_sm, old.wave_paths)
    (a, (_, a2, an)), (b, (_, b2, bn)) = films
    assert np.array_equal(an, bn) and (an == 3).all()
    assert np.allclose(a, b, rtol=1e-6, atol=1e-7)
    assert np.allclose(a2, b2, rtol=1e-6, atol=1e-9)


@pytest.mark.parametrize("size", [(1, 1), (31, 1), (33, 1), (511, 1), (19, 27), (1025, 1)])
def test_smallest_films(gpu_ctx, size):
    w, h = size
    sd = S.cornell(w, h, spp=1)
    sc = G.Scene(gpu_ctx, sd, A.BG_BVH_WIDE)
    r = G.PathIntegrator(sd.camera, 1, 5).render(sc)
    assert r.stats.error_word == 0
    _, _, n = G.PathIntegrator.moments(gpu_ctx, w, h)
    assert (n == 1).all()


@pytest.mark.parametrize("mode", [A.BG_MODE_REF_COMPAT, A.BG_MODE_PBRT])
@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (33, 1, 1), (1023, 1, 1), (1025, 1, 3), (400, 401, 1)])
def test_per_path_kernel_films(gpu_ctx, mode, w, h, spp):
    """Reference layout: fewer paths than a block, than the grid, and more (threads start further
    paths).  Every sample reaches the film once, and the film equals the oracle's: same paths and
    operations without contraction, so all but a few channels are equal to 1e-5 (transcendental
    functions of the two machines differ in their last bits)."""
    import oracle as O
    sd = S.cornell(w, h, spp=spp)
    sc = G.Scene(gpu_ctx, sd, A.BG_BVH_REFERENCE)
    r = G.PathIntegrator(sd.camera, spp, 5, mode=mode).render(sc)
    assert r.stats.error_word == 0
    _, _, n = G.PathIntegrator.moments(gpu_ctx, w, h)
    assert (n == spp).all()
    ref = O.OracleScene(sd, fixed_bvh=False).render(mode)["rgb"]
    assert np.mean(np.abs(r.rgb - ref) <= 1e-5 * (1.0 + np.abs(ref))) >= 0.99
