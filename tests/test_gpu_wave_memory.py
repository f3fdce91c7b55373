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
