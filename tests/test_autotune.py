"""The autotuner's choices, with the engine and its timings replaced by stand-ins (no GPU)."""
import json
from types import SimpleNamespace

import pytest


class _Lib:
    def __init__(self, log):
        self.log = log

    def spi_set_kernel_for(self, h, population, layout, min_blocks):
        self.log.append((bool(population), layout, min_blocks))
        return 0


def _engine(population, log, torque_speed=1):
    return SimpleNamespace(lib=_Lib(log), _h=None, device=None, stream=None, N=64, W=8, H=5, population=population, variant="lane3",
                           _robot=SimpleNamespace(torque_speed=torque_speed, motor_gain=(1.0, 1.0, 1.0), tanh_a=(0.0, 0.0, 0.0)))


@pytest.fixture
def tuner(monkeypatch, tmp_path):
    from spi_gb300 import autotune
    monkeypatch.setattr(autotune.torch.cuda, "get_device_name", lambda d: "GPU")
    monkeypatch.setattr(autotune, "CACHE", tmp_path / "autotune.json")
    # a caller's batch: the lane variants are one kernel, told apart by noise only; a population: quad4 ahead
    ms = {False: dict(quad3=2.0, quad4=2.0, quad5=2.0, lane2=0.995, lane3=1.0, lane4=0.99, block3=3.0, block4=3.0, block5=3.0),
          True: dict(quad3=1.1, quad4=1.0, quad5=1.2, lane2=3.0, lane3=2.0, lane4=2.1, block3=1.3, block4=1.3, block5=1.3)}
    calls = []

    def time(engine, population, reps):
        last = [c for c in engine.lib.log if c[0] == population][-1]
        calls.append((population, last))
        return ms[population][next(n for n, lay, mb in autotune.VARIANTS if (lay, mb) == last[1:])]
    monkeypatch.setattr(autotune, "_time", time)
    return SimpleNamespace(mod=autotune, calls=calls, cache=tmp_path / "autotune.json")


def test_tuning_a_callers_batch_tunes_the_cem_apart(tuner):
    log = []
    e = _engine(False, log)
    best, times = tuner.mod.tune_engine(e)
    assert best == e.variant == "lane3" and times["lane4"] == 0.99
    assert [c for c in log if c[0]][-1] == (True, 0, 4) and [c for c in log if not c[0]][-1] == (False, 1, 3)


def test_tuning_a_population_leaves_the_callers_kernel(tuner):
    log = []
    best, _ = tuner.mod.tune_engine(_engine(True, log))
    assert best == "quad4" and all(c[0] for c in log)


def test_cached_choices_are_of_the_same_batch_motor_and_build(tuner, monkeypatch, tmp_path):
    tuner.mod.tune_engine(_engine(True, []))
    n = len(tuner.calls)
    tuner.mod.tune_engine(_engine(True, []))
    assert len(tuner.calls) == n                                  # the same: from the cache
    tuner.mod.tune_engine(_engine(True, [], torque_speed=0))
    assert len(tuner.calls) == 2 * n                              # another motor shape
    tuner.mod.tune_engine(_engine(False, []))
    assert len(tuner.calls) == 3 * n                              # a caller's batch: its own, the population's cached
    monkeypatch.setattr(tuner.mod, "LIB_DIR", tmp_path)
    (tmp_path / ".stamp").write_text("another build")
    tuner.mod.tune_engine(_engine(True, []))
    assert len(tuner.calls) == 4 * n and len(json.loads(tuner.cache.read_text())) == 4
