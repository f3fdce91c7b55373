"""Launches that may start while the previous one ends.  A stage that read before its predecessor had
written would change the film, so renders are compared bit for bit with the same render under stage
timing, whose events between the launches keep them apart: films of a pixel, around a warp and around
the blocks of the stages, one and several material classes, the ray-binning stage, and several waves."""
import numpy as np
import pytest

from bonsai_gb300 import _abi as A
from bonsai_gb300 import autotune
from bonsai_gb300 import gpu as G
from bonsai_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,layout", [("cornell", A.BG_BVH_WIDE), ("cornell", A.BG_BVH_WIDE2),
                                         ("textured", A.BG_BVH_WIDE)])
@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (33, 1, 1), (127, 5, 2), (64, 64, 1), (257, 129, 3)])
@pytest.mark.parametrize("sort,wave", [(0, 1 << 20), (1, 1 << 20), (0, 1025)])
def test_same_film_as_separate_launches(gpu_ctx, kind, layout, w, h, spp, sort, wave):
    sd = (S.textured_room if kind == "textured" else S.cornell)(w, h, spp=spp)
    sc = G.Scene(gpu_ctx, sd, layout)
    integ = G.PathIntegrator(sd.camera, spp, 5)
    old = autotune.get(gpu_ctx)
    try:
        autotune.set_(gpu_ctx, old.refill, old.blocks_per_sm, wave, sort)
        apart = integ.render(sc, stage_timing=True).rgb
        for graph in (False, False, False, True, True):
            r = integ.render(sc, graph=graph)
            assert r.stats.error_word == 0
            assert np.array_equal(r.rgb, apart)
    finally:
        autotune.set_(gpu_ctx, old.refill, old.blocks_per_sm, old.wave_paths)


@pytest.mark.parametrize("integrator", ["whitted", "direct"])
@pytest.mark.parametrize("layout", [A.BG_BVH_WIDE, A.BG_BVH_WIDE2])
@pytest.mark.parametrize("w,h,spp,depth", [(1, 1, 1, 1), (33, 1, 1, 2), (127, 5, 2, 5), (64, 64, 1, 8)])
def test_tree_levels_equal_the_per_thread_kernel(gpu_ctx, integrator, layout, w, h, spp, depth):
    """The tree wavefront's levels against one thread per sample over the reference layout: the same
    trees; the sums differ in order and contraction, so all but a few channels (hits of rays at an
    edge, 1e-2 of them at the most) are equal to 1e-4 of their size."""
    sd = S.cornell(w, h, spp=spp)
    integ = {"whitted": lambda: G.WhittedIntegrator(sd.camera, spp, depth),
             "direct": lambda: G.DirectLightingIntegrator(sd.camera, spp, depth)}[integrator]()
    ref = integ.render(G.Scene(gpu_ctx, sd, A.BG_BVH_REFERENCE)).rgb
    sc = G.Scene(gpu_ctx, sd, layout)
    for _ in range(3):
        r = integ.render(sc)
        assert r.stats.error_word == 0
        assert np.mean(np.abs(r.rgb - ref) <= 1e-4 * (1.0 + np.abs(ref))) >= 0.99
