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
