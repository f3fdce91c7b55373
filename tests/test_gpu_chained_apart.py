"""Chained launches against launches that are not chained.

A batch's stages are launched plainly, one after the end of the other, so a batch of one scene is the arm in
which no stage can start early; the path wavefront chains generation, extension, binning and the shadow
rays' successor.  A stage that read before its predecessor had written would lose or repeat paths.  The two
are different kernels (the batch's look a path's scene up), so films are compared as same paths.

The graph of a context that has rendered nothing larger replays its launches for every wave: bit for bit the
plain waves' film."""
import numpy as np
import pytest

from bonsai_gb300 import _abi as A
from bonsai_gb300 import autotune
from bonsai_gb300 import gpu as G
from bonsai_gb300 import scenes as S
from .parity import assert_same_paths

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["cornell", "textured"])
@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (33, 1, 1), (127, 5, 2), (64, 64, 1), (257, 129, 3)])
@pytest.mark.parametrize("sort,wave", [(0, 1 << 20), (1, 1 << 20), (0, 1025)])
def test_same_film_as_a_batch_of_one(gpu_ctx, kind, w, h, spp, sort, wave):
    sd = (S.textured_room if kind == "textured" else S.cornell)(w, h, spp=spp)
    sc = G.Scene(gpu_ctx, sd, A.BG_BVH_WIDE)
    it = G.PathIntegrator(sd.camera, spp, 5, seed=2)
    old = autotune.get(gpu_ctx)
    try:
        autotune.set_(gpu_ctx, old.refill, old.blocks_per_sm, 1 << 20)
        (apart,), _ = G.render_batch(gpu_ctx, [G.BatchJob(sc, sd.camera, spp, 5, seed=2)])
        n0 = G.PathIntegrator.moments(gpu_ctx, w * h, 1)[2].reshape(h, w)
        autotune.set_(gpu_ctx, old.refill, old.blocks_per_sm, wave, sort)
        for graph in (False, False, True, True):
            r = it.render(sc, graph=graph)
            assert r.stats.error_word == 0
            n = G.PathIntegrator.moments(gpu_ctx, w, h)[2]
            assert np.array_equal(n, n0) and (n == spp).all()
            assert_same_paths(r.rgb, apart)
    finally:
        autotune.set_(gpu_ctx, old.refill, old.blocks_per_sm, old.wave_paths)
        sc.close()


@pytest.mark.parametrize("w,h,spp", [(127, 5, 2), (257, 129, 3)])
def test_graph_of_several_waves(w, h, spp):
    sd = S.cornell(w, h, spp=spp)
    ctx = G.Context(0, max_queue_paths=1025)  # nothing in it holds more than 1025 paths
    try:
        sc = G.Scene(ctx, sd, A.BG_BVH_WIDE)
        it = G.PathIntegrator(sd.camera, spp, 5)
        plain = it.render(sc)
        for _ in range(3):
            r = it.render(sc, graph=True)
            assert r.stats.error_word == 0
            assert r.stats.extension_rays == plain.stats.extension_rays
            assert np.array_equal(r.rgb, plain.rgb)
    finally:
        ctx.close()
