"""What an engine holds between calls: its theta batch, its CEM and the captured CEM step."""
import numpy as np
import pytest
import torch

from helpers import oracle_windows, random_theta
from oracle import go2_model as gm

pytestmark = pytest.mark.gpu


def _engine(windows):
    from spi_gb300.engine import Engine
    e = Engine()
    e.load_windows(*windows)
    return e


def _windows(W, H=3):
    _, init, actions, target = oracle_windows(60, n_traj=2, T=40, H=H)
    return [torch.from_numpy(a[:W]) for a in (init, actions, target)]


def _cem(e, n=64):
    from spi_gb300.cem import CEM
    return CEM(e, n_samples=n, param_ids=[0, 4], lo=gm.THETA_PRIOR_LO[[0, 4]], hi=gm.THETA_PRIOR_HI[[0, 4]],
               nominal=gm.THETA_NOMINAL, seed=5)


@pytest.mark.parametrize("graph", [True, False])
def test_evaluation_between_cem_runs(built, graph):
    """After the second CEM run the batch is the population again, in its size and its kernel: population and
    costs are those of a CEM with no evaluation in between, to the bit."""
    windows, got = _windows(19), []
    for th in (None, random_theta(np.random.default_rng(1), 16).astype(np.float32)):
        e = _engine(windows)
        cem = _cem(e)
        cem.run(2, graph=graph)
        if th is not None:
            e.evaluate(torch.from_numpy(th))
        cem.run(1, graph=graph)
        pop, costs = cem.theta(), e.read()[1]
        e.run()
        got.append((pop, costs, e.read()[1], cem.read()))
    a, b = got
    assert a[0].shape == (64, 13) and all(torch.equal(x, y) for x, y in zip(a[:3], b[:3]))
    assert torch.equal(a[1], a[2])
    assert a[3]["best_cost"] == b[3]["best_cost"] and np.array_equal(a[3]["mu"], b[3]["mu"])


def _too_many(W):
    """Theta samples whose window-group results (36 bytes each) no GPU holds: 300,000 of 32,768 groups, 354 GB."""
    assert W == 32768 * 8
    return torch.from_numpy(random_theta(np.random.default_rng(2), 300).astype(np.float32)).repeat(1000, 1)


def _many_windows():
    w = [a[:1].repeat(32768 * 8, *([1] * (a.ndim - 1))) for a in _windows(19, H=1)]
    return w


def test_evaluation_without_memory_leaves_the_batch(built):
    """An evaluation that finds no memory fails as spi_set_theta and a failing spi_run do: the batch is the caller's,
    and runs once the windows are fewer."""
    from spi_gb300 import _lib
    few, th = _windows(8, H=1), _too_many(32768 * 8)
    e = _engine(_many_windows())
    e.evaluate(th[:2])
    with pytest.raises(_lib.SpiError) as err:
        e.evaluate(th)
    assert err.value.code == _lib.SPI_ENOMEM
    with pytest.raises(_lib.SpiError):
        e.read()
    e.load_windows(*few)
    e.run()
    cost = e.read()[1]
    assert cost.shape == (300000,) and torch.equal(cost, _engine(few).evaluate(th)[1])


def test_cem_after_an_evaluation_without_memory(built):
    """The failed evaluation has moved buffers that the captured CEM step refers to; the next run is still that of a
    CEM without it, to the bit."""
    from spi_gb300 import _lib
    windows, got = _many_windows(), []
    for fail in (False, True):
        e = _engine(windows)
        cem = _cem(e, n=4)
        cem.run(2)
        if fail:
            with pytest.raises(_lib.SpiError):
                e.evaluate(_too_many(32768 * 8))
        cem.run(1)
        got.append((cem.theta(), e.read()[1], cem.read()["best_cost"]))
        e.close()
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1]) and got[0][2] == got[1][2]


@pytest.mark.parametrize("variant", ["lane2", "lane3", "quad4"])
def test_a_callers_batch_by_the_populations_kernels(built, variant):
    """The CEM's theta samples set by the caller and run as a population: the CEM's costs, to the bit; its own choice of
    kernel leaves the other's alone."""
    from spi_gb300 import _lib
    from spi_gb300.autotune import _BY_NAME, set_variant
    windows = _windows(19)
    e, other = _engine(windows), _engine(windows)
    set_variant(e, "lane3")
    _, layout, min_blocks = _BY_NAME[variant]
    for x in (e, other):
        _lib.check(x.lib.spi_set_kernel_for(x._h, 1, layout, min_blocks))
    cem = _cem(e)
    cem.sample()
    th = cem.theta()
    e.run()
    comp, cost = e.read()
    other.set_theta(th)
    other.run(population=True)
    c, v = other.read()
    assert torch.equal(c, comp) and torch.equal(v, cost)
    plain = _engine(windows).evaluate(th)[1]
    assert torch.equal(other.evaluate(th)[1], plain)


def test_tuning_keeps_a_choice_for_each_batch(built, monkeypatch, tmp_path):
    from spi_gb300 import autotune
    monkeypatch.setattr(autotune, "CACHE", tmp_path / "autotune.json")
    e = _engine(_windows(19))
    e.evaluate(torch.from_numpy(random_theta(np.random.default_rng(4), 64).astype(np.float32)))
    best, ms = autotune.tune_engine(e)
    assert best in ms and set(ms) == {v[0] for v in autotune.VARIANTS}
    cem = _cem(e)
    cem.run(2)
    assert np.isfinite(cem.read()["best_cost"])
    assert autotune.tune_engine(e)[0] in ms
