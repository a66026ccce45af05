"""Kernel-variant autotuner for the rollout kernel.

The rollout kernel comes in three lane layouts -- "quad" (four lanes per rollout, one leg
each), "block" (the quad layout with each rollout's base solved once by one warp of the CTA)
and "lane" (one lane per rollout through all four legs) -- and occupancy variants: the
register allocator targets 2..5 CTAs of 128 threads per SM (255 / 168 / 128 / 96 registers
per thread, with more spilling as registers shrink). Which is fastest depends on the
horizon, the window count and the GPU, so the variant is picked by timing each on the caller's
own windows and theta batch, apart for a caller's batch and a CEM's population. Choices are cached per (GPU,
horizon bucket, work bucket, window-count remainder, whose batch, motor shape, build) in the build folder.
"""
from __future__ import annotations

import json
import math
from pathlib import Path

import torch

from . import _lib
from ._build import LIB_DIR

CACHE = LIB_DIR / "autotune.json"
# (name, layout, min_blocks); layout 0 = SPI_LAYOUT_QUAD, 1 = SPI_LAYOUT_LANE, 2 = SPI_LAYOUT_BLOCK
VARIANTS = (("quad3", 0, 3), ("quad4", 0, 4), ("quad5", 0, 5), ("lane2", 1, 2), ("lane3", 1, 3), ("lane4", 1, 4),
            ("block3", 2, 3), ("block4", 2, 4), ("block5", 2, 5))
_BY_NAME = {v[0]: v for v in VARIANTS}


DEFAULT = "lane3"


def _key(engine, population):
    """GPU, sizes, motor shape, whose batch and which build a choice was timed with."""
    name = torch.cuda.get_device_name(engine.device).replace(" ", "_")
    work = engine.N * ((engine.W + 7) // 8)
    r = engine._robot
    plain = bool(r.torque_speed) and all(g == 1.0 for g in r.motor_gain) and all(a == 0.0 for a in r.tanh_a)
    stamp = LIB_DIR / ".stamp"
    build = stamp.read_text()[:12] if stamp.exists() else ""
    return (f"{name}|H{2 ** max(0, math.ceil(math.log2(max(engine.H, 1))))}"
            f"|G{2 ** max(0, math.ceil(math.log2(max(work, 1))))}|W%32={engine.W % 32}"
            f"|{'population' if population else 'batch'}|{'speed limit' if plain else 'run-time motor'}|{build}")


def _load():
    try:
        return json.loads(Path(CACHE).read_text())
    except (OSError, ValueError):
        return {}


def set_variant(engine, name):
    """Select a rollout-kernel variant by name (one of VARIANTS)."""
    _, layout, min_blocks = _BY_NAME[name]
    _lib.check(engine.lib.spi_set_kernel_layout(engine._h, int(layout)))
    _lib.check(engine.lib.spi_set_kernel_config(engine._h, int(min_blocks)))
    engine.variant = name


def _set_for(engine, population, name):
    _, layout, min_blocks = _BY_NAME[name]
    _lib.check(engine.lib.spi_set_kernel_for(engine._h, int(population), int(layout), int(min_blocks)))


def _time(engine, population, reps):
    """ms of a rollout launch with the current variant of a caller's batch or of a CEM's population."""
    run = (lambda: engine.run(population=True)) if population else engine.run
    run()
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    t0.record(engine.stream)
    for _ in range(reps):
        run()
    t1.record(engine.stream)
    t1.synchronize()
    return t0.elapsed_time(t1) / reps


def _pick(times, population):
    """The fastest; of a caller's batch the default if it is within 2 % of it: below some size its lane variants are
    one kernel, and which of them a timing favours is noise that a larger batch would pay for."""
    best = min(times, key=times.get)
    return DEFAULT if not population and times[DEFAULT] <= 1.02 * times[best] else best


def tune_engine(engine, reps=3, use_cache=True):
    """Time every variant on the engine's loaded windows and theta batch; keep the fastest.

    A caller's batch (``set_theta``) and a CEM's population take kernels of their own. On a caller's batch both
    are timed and each keeps its fastest, so that a CEM on the engine afterwards is tuned as well; on a
    population its own. Returns (chosen variant, {variant: ms per launch}) of the loaded batch.
    """
    cache = _load() if use_cache else {}
    kinds = (True,) if engine.population else (True, False)     # the loaded batch's own last
    for population in kinds:
        key = _key(engine, population)
        if not (use_cache and key in cache and cache[key]["best"] in _BY_NAME):
            times = {}
            for name, _, _ in VARIANTS:
                _set_for(engine, population, name)
                times[name] = _time(engine, population, reps)
            cache[key] = {"best": _pick(times, population), "ms": times}
        best, times = cache[key]["best"], cache[key]["ms"]
        _set_for(engine, population, best)
    engine.variant = best
    try:
        LIB_DIR.mkdir(exist_ok=True)
        Path(CACHE).write_text(json.dumps(cache, indent=1))
    except OSError:
        pass
    return best, times
