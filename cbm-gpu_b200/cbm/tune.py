"""Autotuner for a plan's launch knobs (row-split threshold, claim sizes, kernel
variant, team size, L2 retention).

``autotune(plan, op, x, y)`` times each candidate configuration on the actual
operands with CUDA events (after warm-up, each candidate the median of a few
repetitions), leaves the plan tuned to the fastest and returns the timings.
Results are remembered per (plan, op, columns, dtypes), so a second call with
the same shapes only re-applies the winner.  Re-laying out a plan (a new
chunk size or hot set) is host work: tune before capturing CUDA graphs.
"""
from __future__ import annotations

import itertools
import statistics

import torch

__all__ = ["autotune", "candidates", "DEFAULT_SPACE"]

DEFAULT_SPACE = {
    "chunk_nnz": [128, 256, 512],
    "rows_per_claim": [2, 4, 8],
    "variant": ["register", "staged"],
    "hot_rows": [0, 65536],
}

# what the register kernel does not read: it claims one group of rows at a time or
# two ahead by itself, has its own team sizes and no L2 hints
_STAGED_ONLY = ("rows_per_claim", "rows_per_claim_deep", "hot_rows", "team")

_cache = {}


def _product(space):
    return [dict(zip(space, values)) for values in itertools.product(*space.values())]


def candidates(space):
    """The configurations of a space, those of the register kernel without the knobs
    that it does not read (they keep the first value listed)."""
    out = []
    for cfg in _product(space):
        if cfg.get("variant") == "register":
            cfg.update({k: space[k][0] for k in _STAGED_ONLY if k in cfg})
        if cfg not in out:
            out.append(cfg)
    return out


def _time(fn, reps, iters):
    ts = []
    for _ in range(reps):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(iters):
            fn()
        e1.record()
        torch.cuda.synchronize()
        ts.append(e0.elapsed_time(e1) / iters)
    return statistics.median(ts)


def autotune(plan, op, x, y, space=None, reps=3, iters=5, warmup=2):
    """Tunes ``plan`` for y <- op(A) x; returns [(config, ms)] sorted by time.
    ``space``: the values to try of each knob, all combinations of them, or a list of
    configurations (default: the ``candidates`` of DEFAULT_SPACE)."""
    key = (id(plan), op, x.shape[1], x.dtype, y.dtype)
    if key in _cache:
        best = _cache[key][0][0]
        plan.tune(**best)
        return _cache[key]
    space = candidates(DEFAULT_SPACE) if space is None else _product(space) if isinstance(space, dict) else space
    results = []
    for cfg in space:
        plan.tune(**cfg)
        fn = lambda: plan.matmul(op, x, y)  # noqa: E731
        for _ in range(warmup):
            fn()
        torch.cuda.synchronize()
        results.append((cfg, _time(fn, reps, iters)))
    results.sort(key=lambda r: r[1])
    plan.tune(**results[0][0])
    plan.check_device()
    _cache[key] = results
    return results
