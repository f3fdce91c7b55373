"""Paths per wave and the device memory that they take: a caller's own size is taken as it is.

The number of a render's kernel launches tells the number of its waves (both films below take the same
launches a wave)."""
import numpy as np
import pytest

from bonsai_gb300 import _abi as A
from bonsai_gb300 import autotune
from bonsai_gb300 import gpu as G
from bonsai_gb300 import scenes as S

pytestmark = pytest.mark.gpu

LARGEST = 1 << 25  # the library's own choice without a memory cap, 8.1 GB


def _set_wave(ctx, wave):
    t = autotune.get(ctx)
    autotune.set_(ctx, t.refill, t.blocks_per_sm, wave)


def _launches(ctx, paths):
    """Launches of a render of `paths` paths, and of one of a single pixel (one wave)."""
    out = []
    for w, h, spp in ((1024, paths // (1024 * 8), 8), (1, 1, 1)):
        sd = S.cornell(w, h)
        sc = G.Scene(ctx, sd, A.BG_BVH_WIDE)
        out.append(G.PathIntegrator(sd.camera, spp, 3).render(sc, readback=False).stats.launches)
        sc.close()
    return out


def test_callers_wave_size_under_a_memory_cap():
    cap = 12 << 30
    ctx = G.Context(0, memory_cap_bytes=cap)
    try:
        assert autotune.get(ctx).wave_paths == 1 << 22  # the library's choice under a cap
        many, one = _launches(ctx, 1 << 23)
        assert many - 1 == 2 * (one - 1)  # two waves, and the launch that resolves the film
        _set_wave(ctx, LARGEST)
        assert autotune.get(ctx).wave_paths == LARGEST
        many, one = _launches(ctx, 1 << 23)
        assert many == one
    finally:
        ctx.close()
    ctx = G.Context(0, max_queue_paths=LARGEST, memory_cap_bytes=cap)
    try:
        assert autotune.get(ctx).wave_paths == LARGEST
        many, one = _launches(ctx, 1 << 23)
        assert many == one
    finally:
        ctx.close()


def test_callers_wave_size_beyond_the_cap_is_refused():
    ctx = G.Context(0, memory_cap_bytes=2 << 30)
    try:
        _set_wave(ctx, LARGEST)
        with pytest.raises(G.BonsaiError) as ei:
            _launches(ctx, LARGEST)
        assert ei.value.status == A.BG_ERR_OOM
        _set_wave(ctx, 1 << 20)  # the context stays usable
        _launches(ctx, 1 << 21)
    finally:
        ctx.close()


def test_callers_wave_size_in_a_guided_render(gpu_ctx):
    """A film of more than 2^22 pixels: the library's choice for guided renders is 2^22 paths a wave."""
    sd = S.cornell(2200, 2000)
    launches = []
    for wave in (0, LARGEST):
        ctx = G.Context(0, max_queue_paths=wave)
        try:
            sc = G.Scene(ctx, sd, A.BG_BVH_WIDE)
            g = G.Guide(ctx, warmup_passes=100, no_train=True, no_fallback=True)
            r = G.PathIntegrator(sd.camera, 1, 3).render_guided(sc, g, readback=False)
            launches.append(r.stats.launches)
        finally:
            ctx.close()
    # a guided call's launches outside its waves: the relative variance and the film's resolution
    assert launches[0] - 2 == 2 * (launches[1] - 2)


def test_setting_what_get_says_changes_nothing(gpu_ctx):
    ctx = G.Context(0)
    try:
        sd = S.cornell(64, 64, spp=2)
        sc = G.Scene(ctx, sd, A.BG_BVH_WIDE)
        a = G.PathIntegrator(sd.camera, 2, 4).render(sc)
        t = autotune.get(ctx)
        assert t.wave_paths == LARGEST
        _set_wave(ctx, t.wave_paths)
        b = G.PathIntegrator(sd.camera, 2, 4).render(sc)
        assert autotune.get(ctx).wave_paths == LARGEST
        assert np.array_equal(a.rgb, b.rgb) and a.stats.launches == b.stats.launches
    finally:
        ctx.close()


def _free():
    import torch
    return torch.cuda.mem_get_info()[0]


def _film(ctx, spp=32):
    """A film of 2^20 pixels: 2^25 paths at 32 samples."""
    sd = S.cornell(1024, 1024)
    sc = G.Scene(ctx, sd, A.BG_BVH_WIDE)
    try:
        return G.PathIntegrator(sd.camera, spp, 3).render(sc).rgb
    finally:
        sc.close()


def test_a_large_wave_makes_way_for_other_allocations():
    """More than is free with the 8.1 GB wave, less than is free without it: the same context's next allocation
    succeeds, and renders go on."""
    ctx = G.Context(0)
    try:
        before = _free()
        want = _film(ctx)
        held = before - _free()
        if held < 7 << 30:
            pytest.skip("the device has too little free memory for the largest wave")
        p = ctx.alloc(_free() + (4 << 30))
        assert _free() > 1 << 30
        ctx.free(p)
        assert before - _free() < 1 << 30  # scene, film: the wave is gone
        assert np.array_equal(_film(ctx), want)  # and comes back
        assert before - _free() >= held - (1 << 28)
    finally:
        ctx.close()


def test_a_wave_takes_a_share_of_the_free_memory():
    """With 60 GB free a wave is at most 60 / 16 GB (2^23 paths, 2.0 GB), with 10 GB free 2^22 paths (1.0 GB), as
    on a device with plenty the film is the same samples."""
    other = G.Context(0)
    plenty = G.Context(0)
    try:
        if _free() < 200 << 30:
            pytest.skip("needs most of the device free")
        want = _film(plenty)
        plenty.close()
        for leave, most in ((60 << 30, 60 << 26), (10 << 30, 240 << 22)):
            p = other.alloc(_free() - leave)
            ctx = G.Context(0)
            try:
                before = _free()
                got = _film(ctx)
                took = before - _free() - 64 * (1 << 20)  # less the film
                assert took <= most + (64 << 20), (leave, took)
                np.testing.assert_allclose(got, want, rtol=1e-6, atol=0)
            finally:
                ctx.close()
                other.free(p)
    finally:
        other.close()
