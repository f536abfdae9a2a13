"""Autotuner host logic on the CPU: the fastest built variant is kept,
variants a Riemann solver was not built with are skipped, other errors
propagate, and the per-workload JSON cache short-cuts later trials.  The
batch is a stand-in that returns fixed timings (no device call)."""
import json

import pytest

from bonzo_b200 import _lib, autotune


class FakeBatch:
    def __init__(self, ms, unsupported=(), fail=None):
        self.ms, self.unsupported, self.fail = ms, set(unsupported), fail
        self.timed, self.chosen = [], None

    def time_variant(self, v, steps):
        self.timed.append(v)
        if v == self.fail:
            raise _lib.BnzError(_lib.BNZ_ERR_CUDA, "launch failed")
        if v in self.unsupported:
            raise _lib.BnzError(_lib.BNZ_ERR_UNSUPPORTED, "not built")
        return self.ms[v]

    def set_variant(self, v):
        self.chosen = v


@pytest.fixture
def cache(tmp_path, monkeypatch):
    p = tmp_path / "tune.json"
    monkeypatch.setenv("BNZ_TUNE_CACHE", str(p))
    return p


def _timings(nv):
    return {v: 10.0 - 0.5 * ((v * 7) % nv) for v in range(nv)}


def test_workload_key_buckets():
    assert autotune.workload_key([128] * 64, "hlld", "vl") == "2d|hlld|vl|inst=6|meanN=7"
    # sweeps of similar shape share a bucket
    assert (autotune.workload_key([120, 136] * 32, "hlld", "vl")
            == autotune.workload_key([128] * 64, "hlld", "vl"))
    assert autotune.workload_key([128] * 64, "hll", "mc") != autotune.workload_key([128] * 64, "hlld", "mc")


def test_fastest_variant_kept_and_cached(cache):
    nv = len(_lib.variants())
    ms = _timings(nv)
    b = FakeBatch(ms)
    best, t = autotune.tune_batch(b, [64] * 8, steps=1)
    assert best == min(ms, key=ms.get) and b.chosen == best
    assert b.timed == list(range(nv)) and t == ms
    d = json.loads(cache.read_text())
    key = autotune.workload_key([64] * 8, "hlld", "vl")
    assert d[key]["variant"] == best and len(d[key]["variants"]) == nv
    # a second sweep of the same shape reads the cache and times nothing
    b2 = FakeBatch(ms)
    best2, t2 = autotune.tune_batch(b2, [64] * 8, steps=1)
    assert best2 == best and b2.chosen == best and b2.timed == [] and t2 == ms


def test_cached_choice_is_for_the_same_kernels(cache):
    """A choice timed without the strip walks (another batch, an older library)
    does not answer for a batch that can walk, nor the reverse."""
    nv = len(_lib.variants())
    ms = _timings(nv)
    autotune.tune_batch(FakeBatch(ms), [64] * 8)
    b = FakeBatch({**ms, _lib.WALK_VARIANT: 0.1})
    b.walk_variant = _lib.WALK_VARIANT
    best, t = autotune.tune_batch(b, [64] * 8)
    assert best == b.chosen == _lib.WALK_VARIANT and b.timed == list(range(nv)) + [_lib.WALK_VARIANT]
    assert autotune.tune_batch(b, [64] * 8)[0] == _lib.WALK_VARIANT and len(b.timed) == nv + 1  # cached
    b2 = FakeBatch(ms)
    assert autotune.tune_batch(b2, [64] * 8)[0] == min(ms, key=ms.get) and len(b2.timed) == nv
    d = json.loads(cache.read_text())
    for e in d.values():
        del e["variants"]
    cache.write_text(json.dumps(d))
    b3 = FakeBatch(ms)
    autotune.tune_batch(b3, [64] * 8)
    assert len(b3.timed) == nv


def test_workload_key_tells_zones_and_slopes_apart():
    even, uneven = [128] * 64, [16] * 48 + [464] * 16  # the same number of grids and mean side
    assert autotune.workload_key(even, "hlld", "vl") != autotune.workload_key(uneven, "hlld", "vl")
    assert autotune.workload_key(even, "hlld", "vl") != autotune.workload_key(even, "hlld", "vl", charact_proj=True)


def test_variant_names():
    names = [_lib.variant_name(v) for v in range(len(_lib.variants()) + 1)]
    assert names[_lib.WALK_VARIANT] == "walk" and names[8] == "15x14pp" and len(set(names)) == len(names)


def test_unsupported_variants_skipped(cache):
    nv = len(_lib.variants())
    ms = _timings(nv)
    fastest = min(ms, key=ms.get)
    b = FakeBatch(ms, unsupported=[fastest])
    best, t = autotune.tune_batch(b, [64] * 8, rsolver="hll", use_cache=False)
    assert fastest not in t and best != fastest and best == min(t, key=t.get)
    assert not cache.exists()


def test_other_errors_propagate(cache):
    nv = len(_lib.variants())
    b = FakeBatch(_timings(nv), fail=1)
    with pytest.raises(_lib.BnzError) as e:
        autotune.tune_batch(b, [64] * 8)
    assert e.value.code == _lib.BNZ_ERR_CUDA
    assert b.chosen is None and not cache.exists()


def test_unreadable_cache_ignored(cache):
    cache.write_text("{not json")
    nv = len(_lib.variants())
    b = FakeBatch(_timings(nv))
    best, _ = autotune.tune_batch(b, [64] * 8)
    assert b.chosen == best and len(b.timed) == nv
    assert json.loads(cache.read_text())  # rewritten whole
