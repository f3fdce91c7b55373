"""Films of few pixels and many samples: several threads share a pixel in the film pass.

Every sample must reach its pixel once.  The other arm renders the same samples in accumulated pieces of
255 a pixel, where one thread adds a pixel's samples: the same paths, so FP64 sums of at most 70,000
non-negative terms in another order, equal to 70,000 * 2^-53 = 8e-12 (1e-11 here)."""
import ctypes as C

import numpy as np
import pytest

from bonsai_gb300 import _abi as A
from bonsai_gb300 import autotune
from bonsai_gb300 import gpu as G
from bonsai_gb300 import scenes as S

pytestmark = pytest.mark.gpu

PIECE = 255


def _pieces(ctx, sc, camera, spp, depth, seed=0):
    for s0 in range(0, spp, PIECE):
        G.PathIntegrator(camera, min(PIECE, spp - s0), depth, seed=seed).render(sc, first_sample=s0, accumulate=s0 > 0)
    return G.PathIntegrator.moments(ctx, camera.width, camera.height)


def _same(got, want):
    for g, w in zip(got[:2], want[:2]):
        np.testing.assert_allclose(g, w, rtol=1e-11, atol=0)
    np.testing.assert_array_equal(got[2], want[2])


# one pixel, a row, a remainder of one sample, the edge of the rule (255, 256 samples), several waves, and
# the largest film whose pixels take two threads each
@pytest.mark.parametrize("w,h,spp,wave", [(1, 1, 255, 1 << 20), (1, 1, 256, 1 << 20), (1, 1, 65537, 1 << 20),
                                          (8, 8, 1025, 1 << 20), (33, 3, 1000, 1 << 20), (8, 8, 4097, 70_001),
                                          (1, 1, 65537, 1025), (362, 362, 257, 1 << 26)])
@pytest.mark.parametrize("graph", [False, True])
def test_every_sample_once(gpu_ctx, w, h, spp, wave, graph):
    sd = S.cornell(w, h)
    sc = G.Scene(gpu_ctx, sd, A.BG_BVH_WIDE)
    old = autotune.get(gpu_ctx)
    try:
        autotune.set_(gpu_ctx, old.refill, old.blocks_per_sm, wave)
        r = G.PathIntegrator(sd.camera, spp, 4).render(sc, graph=graph)
        assert r.stats.error_word == 0 and r.stats.samples == w * h * spp
        got = G.PathIntegrator.moments(gpu_ctx, w, h)
        assert (got[2] == spp).all()
        _same(got, _pieces(gpu_ctx, sc, sd.camera, spp, 4))
    finally:
        autotune.set_(gpu_ctx, old.refill, old.blocks_per_sm, old.wave_paths)
        sc.close()


@pytest.mark.parametrize("wave", [1 << 22, 50_021])
def test_batch_of_small_and_ordinary_films(gpu_ctx, wave):
    shapes = [(1, 1, 20_000), (40, 30, 3), (8, 8, 1025), (2, 1, 255), (5, 7, 300)]
    sds = [S.cornell(w, h) for w, h, _ in shapes]
    scenes = [G.Scene(gpu_ctx, sd, A.BG_BVH_WIDE) for sd in sds]
    jobs = [G.BatchJob(sc, sd.camera, spp, 4, seed=9) for sc, sd, (_, _, spp) in zip(scenes, sds, shapes)]
    npix = [w * h for w, h, _ in shapes]
    old = autotune.get(gpu_ctx)
    try:
        autotune.set_(gpu_ctx, old.refill, old.blocks_per_sm, wave)
        _, st = G.render_batch(gpu_ctx, jobs)
        assert st.error_word == 0
        got = G.PathIntegrator.moments(gpu_ctx, sum(npix), 1)
        # the same batch in pieces: the batch's kernels, one thread a pixel
        want = None
        for s0 in range(0, max(s for _, _, s in shapes), PIECE):
            part = [G.BatchJob(sc, sd.camera, max(0, min(PIECE, spp - s0)), 4, seed=9, first_sample=s0)
                    for sc, sd, (_, _, spp) in zip(scenes, sds, shapes)]
            keep = [k for k, p in enumerate(part) if p.spp > 0]
            G.render_batch(gpu_ctx, [part[k] for k in keep])
            m = G.PathIntegrator.moments(gpu_ctx, sum(npix[k] for k in keep), 1)
            if want is None:
                want = tuple(x.copy() for x in m)
                continue
            at = 0
            for k in keep:
                dst = sum(npix[:k])
                for a, b in zip(want, m):
                    a[0, dst:dst + npix[k]] += b[0, at:at + npix[k]]
                at += npix[k]
        _same(got, want)
    finally:
        autotune.set_(gpu_ctx, old.refill, old.blocks_per_sm, old.wave_paths)
        for sc in scenes:
            sc.close()


def test_guided_passes_keep_their_pass_film(gpu_ctx):
    """A guided pass's own sums (its relative variance is computed from them) on a small film."""
    sd = S.cornell(7, 5)
    sc = G.Scene(gpu_ctx, sd, A.BG_BVH_WIDE)
    spp, got = 1200, []
    old = autotune.get(gpu_ctx)
    try:
        for wave in (1 << 20, 35 * PIECE):
            autotune.set_(gpu_ctx, old.refill, old.blocks_per_sm, wave)
            g = G.Guide(gpu_ctx, warmup_passes=100, no_train=True, no_fallback=True, pass_paths=35 * 400)
            r = G.PathIntegrator(sd.camera, spp, 4).render_guided(sc, g)
            assert r.stats.error_word == 0 and r.guide.passes == 3
            got.append((r.guide.relvar_plain, G.PathIntegrator.moments(gpu_ctx, 7, 5)))
            g.close()
        _same(got[0][1], got[1][1])
        # FP32 pass sums of 400 samples: 400 * 2^-24 of the sum, which the variance takes the square of a difference of
        assert abs(got[0][0] - got[1][0]) <= 1e-2 * got[1][0]
    finally:
        autotune.set_(gpu_ctx, old.refill, old.blocks_per_sm, old.wave_paths)
        sc.close()


@pytest.mark.parametrize("w,h,spp", [(1, 1, 70_001), (8, 8, 1025)])  # waves of 65,536 paths: two each
def test_allocation_free_render(gpu_ctx, w, h, spp):
    sd = S.cornell(w, h)
    sc = G.Scene(gpu_ctx, sd, A.BG_BVH_WIDE)
    want = G.PathIntegrator(sd.camera, spp, 4).render(sc).rgb
    cam, o = G.camera_struct(sd.camera), A.bg_render_opts()
    o.spp, o.max_depth, o.rr_threshold, o.mode = spp, 4, 1.0, A.BG_MODE_PBRT
    d_out, got = gpu_ctx.alloc(w * h * 12), np.zeros((h, w, 3), np.float32)
    try:
        gpu_ctx.check(gpu_ctx.lib.bg_render_noalloc(sc.h, C.byref(cam), C.byref(o), d_out, None))
        gpu_ctx.d2h(got, d_out)
    finally:
        gpu_ctx.free(d_out)
        sc.close()
    np.testing.assert_allclose(got, want, rtol=1e-6, atol=0)


def test_few_pixels_take_no_longer_than_many(gpu_ctx):
    """2^20 paths of one pixel against as many of 1024 x 1024 pixels: the same work, but for the sums."""
    ms = []
    for w, spp in ((1, 1 << 20), (16, 1 << 12), (1024, 1)):
        sd = S.cornell(w, w)
        sc = G.Scene(gpu_ctx, sd, A.BG_BVH_WIDE)
        it = G.PathIntegrator(sd.camera, spp, 5)
        it.render(sc)
        ms.append(min(it.render(sc).stats.device_ms for _ in range(3)))
        sc.close()
    assert max(ms[:2]) <= 3.0 * ms[2], ms
