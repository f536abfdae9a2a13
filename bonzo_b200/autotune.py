"""Autotuner for the fused 2D kernels: tile shape, predictor staging, the
persistent kernels and the strip walks.

Every variant the library was built with (bonzo_b200._lib.variants(): tile
tx x ty, shared-memory staging of the predictor's input or not, persistent
work-queue corrector and predictor or not; and the strip walks where the batch
can take them) is timed on
the batch's own state for a few steps (the state is restored after each
trial) and the fastest is kept.  Choices are cached in a JSON file keyed by
the workload shape, so later runs of a similar sweep skip the trials:

    key = "2d|<rsolver>|<limiter>|inst=<log2 bucket>|meanN=<log2 bucket>"

with "|zones=<log2 bucket>" where the two buckets do not give the total of the
zones (sides far from their mean) and "|charact" for characteristic slopes.  An
entry counts only if it was timed over the kernels that the batch has now.

The cache lives at $BNZ_TUNE_CACHE, else ~/.cache/bonzo_b200/fused_tune.json.
"""
import json
import math
import os

from . import _lib

RS_NAME = {v: k for k, v in _lib.RS.items()}
LIM_NAME = {v: k for k, v in _lib.LIM.items()}


def cache_path():
    return os.environ.get("BNZ_TUNE_CACHE",
                          os.path.join(os.path.expanduser("~"), ".cache", "bonzo_b200", "fused_tune.json"))


def workload_key(sizes, rsolver, limiter, charact_proj=False):
    inst, side = round(math.log2(len(sizes))), round(math.log2(sum(sizes) / len(sizes)))
    zones = round(math.log2(sum(n * n for n in sizes)))
    return "2d|%s|%s|inst=%d|meanN=%d%s%s" % (rsolver, limiter, inst, side,
                                             "|zones=%d" % zones if zones != inst + 2 * side else "",
                                             "|charact" if charact_proj else "")


def _load():
    try:
        with open(cache_path()) as f:
            return json.load(f)
    except Exception:
        return {}


def _store(d):
    p = cache_path()
    try:
        os.makedirs(os.path.dirname(p), exist_ok=True)
        tmp = p + ".tmp"
        with open(tmp, "w") as f:
            json.dump(d, f, indent=1, sort_keys=True)
        os.replace(tmp, p)
    except OSError:
        pass  # a read-only home only disables the cache


def tune_batch(batch, sizes, rsolver="hlld", limiter="vl", steps=2, use_cache=True):
    """Pick the fastest variant for `batch` (a bonzo_b200._lib.Batch of grids
    with side lengths `sizes`).  Returns (variant, {variant: ms per step})."""
    key = workload_key(sizes, rsolver, limiter, getattr(batch, "charact_proj", False))
    vs = _lib.variants()
    walk = getattr(batch, "walk_variant", None)
    if use_cache:
        hit = _load().get(key)
        if hit is not None and [tuple(v) for v in hit.get("variants", ())] == vs and hit.get("walk") == walk:
            batch.set_variant(hit["variant"])
            return hit["variant"], {int(k): v for k, v in hit["ms"].items()}
    timings = {}
    for v in list(range(len(vs))) + ([walk] if walk is not None else []):
        try:
            timings[v] = batch.time_variant(v, steps)
        except _lib.BnzError as e:
            if e.code != _lib.BNZ_ERR_UNSUPPORTED:  # not built for this Riemann solver
                raise
    best = min(timings, key=timings.get)
    batch.set_variant(best)
    if use_cache:
        d = _load()
        d[key] = {"variant": best, "ms": timings, "variants": vs, "walk": walk}
        _store(d)
    return best, timings
