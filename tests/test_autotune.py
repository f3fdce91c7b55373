"""The autotuner's cache and descent, with the library's calls faked (no GPU)."""
import json
from types import SimpleNamespace

import pytest

from bonsai_gb300 import _abi as A
from bonsai_gb300 import autotune


@pytest.fixture
def fake(monkeypatch, tmp_path):
    """A context whose renders take a time that the test's `cost` gives; its settings in `now`."""
    lib = tmp_path / "lib.so"
    lib.write_bytes(b"kernels 1")
    f = SimpleNamespace(now=dict(refill=8, blocks_per_sm=8, wave_paths=1 << 25, flags=A.BG_TUNE_CONCURRENT_SHADE), seen=[],
                        cost=lambda cfg: 10.0, lib=lib, cache=tmp_path / "tuning.json")

    def set_(ctx, refill, blocks, wave, sort_rays=0, concurrent_shade=1):
        f.now = dict(refill=refill, blocks_per_sm=blocks, wave_paths=wave,
                     flags=(A.BG_TUNE_SORT_RAYS if sort_rays else 0) | (A.BG_TUNE_CONCURRENT_SHADE if concurrent_shade else 0))

    def trial(ctx, scene, integrator, spp, reps=3):
        f.seen.append(dict(f.now))
        return f.cost(f.now)

    monkeypatch.setattr(autotune, "get", lambda ctx: SimpleNamespace(**f.now))
    monkeypatch.setattr(autotune, "set_", set_)
    monkeypatch.setattr(autotune, "_trial", trial)
    monkeypatch.setattr(autotune, "_gpu_name", lambda: "gpu")
    monkeypatch.setattr(A, "LIB_PATH", lib)
    monkeypatch.setenv("BONSAI_TUNING_CACHE", str(f.cache))
    sd = SimpleNamespace(ntri=12, nsph=0, max_depth=5, camera=SimpleNamespace(width=64, height=64))
    f.tune = lambda **kw: autotune.tune(None, SimpleNamespace(sd=sd), SimpleNamespace(render=lambda *a, **k: None), spp=1, **kw)
    return f


def test_descent_starts_from_the_contexts_settings(fake):
    start = dict(fake.now)
    r = fake.tune()
    assert fake.seen[0] == start
    # nothing is faster: the context's settings stay
    assert (r["refill"], r["blocks_per_sm"], r["wave_paths"], r["sort_rays"], r["concurrent_shade"]) == (8, 8, 1 << 25, 0, 1)
    assert fake.now == start


def test_descent_takes_what_is_faster(fake):
    fake.cost = lambda c: 10.0 - 2.0 * (c["refill"] == 4) - 1.0 * (c["blocks_per_sm"] == 16) - (c["wave_paths"] == 1 << 22)
    r = fake.tune()
    assert (r["refill"], r["blocks_per_sm"], r["wave_paths"]) == (4, 16, 1 << 22) and r["ms"] == 6.0


def test_cache_belongs_to_the_library(fake):
    fake.cost = lambda c: 10.0 - (c["refill"] == 16)
    assert fake.tune()["refill"] == 16
    n = len(fake.seen)
    assert fake.tune()["cached"] and len(fake.seen) == n  # the same library: no trials
    fake.lib.write_bytes(b"kernels 2")
    fake.cost = lambda c: 10.0 - (c["refill"] == 4)
    r = fake.tune()
    assert r["refill"] == 4 and len(fake.seen) > n
    assert len(json.loads(fake.cache.read_text())) == 2
