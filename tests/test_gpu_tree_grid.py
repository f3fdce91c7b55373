"""Tree shading fills the GPU whatever bg_tuning.blocks_per_sm says: the setting is the grid of generation and
traversal.  With 4 blocks of 128 threads per SM instead of 8 traversal loses occupancy only (less than 1.25
times the time in all), with 1 it also loses seven eighths of its threads (3 times at the most); where shading took its
grid from the setting too, it ran on half and on an eighth of the SMs and the renders took 1.4 and 4.5 times
as long.  The films are the same samples: equal to the order of FP32 sums (1e-5)."""
import numpy as np
import pytest

from bonsai_gb300 import _abi as A
from bonsai_gb300 import autotune
from bonsai_gb300 import gpu as G
from bonsai_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cls", [G.DirectLightingIntegrator, G.WhittedIntegrator])
def test_shading_does_not_depend_on_the_traversal_grid(gpu_ctx, cls):
    sd = S.cornell(256, 256)
    sc = G.Scene(gpu_ctx, sd, A.BG_BVH_WIDE)
    it = cls(sd.camera, 16, 5)
    old = autotune.get(gpu_ctx)
    ms, films = {}, {}
    try:
        for blocks in (8, 4, 1, 16):
            autotune.set_(gpu_ctx, old.refill, blocks, old.wave_paths)
            films[blocks] = it.render(sc).rgb
            ms[blocks] = min(it.render(sc).stats.device_ms for _ in range(4))
    finally:
        autotune.set_(gpu_ctx, old.refill, old.blocks_per_sm, old.wave_paths)
        sc.close()
    for blocks in (4, 1, 16):
        np.testing.assert_allclose(films[blocks], films[8], rtol=1e-5, atol=1e-6)
    assert ms[4] <= 1.25 * ms[8] and ms[1] <= 3.0 * ms[8], ms
