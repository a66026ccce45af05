"""The two forms of the evaluation kernel (one lane per rollout, four lanes per rollout) give the
same bits, so the size of a theta batch does not show in its results."""
import numpy as np
import pytest
import torch

from helpers import oracle_windows, random_theta

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [dict(), dict(torque_speed=False), dict(tanh_a=(15.0, 18.0, 25.0), motor_gain=(0.9, 1.1, 1.0))])
@pytest.mark.parametrize("W", [1, 37])
def test_sub_batches_equal_the_full_batch_bit_for_bit(built, W, kw):
    """A batch large enough for the one-lane form (over 12 window groups per SM and theta) and its
    slices from one theta upwards, across the sizes where the four-lane form takes over."""
    from spi_gb300.engine import Engine
    from spi_gb300.robot import SimConfig
    _, init, actions, target = oracle_windows(21, n_traj=2, T=30, H=3)
    e = Engine(SimConfig(**kw))
    e.load_windows(*(torch.from_numpy(a[:W]) for a in (init, actions, target)))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    per = (W + 7) // 8
    n = 60 * sms // per + 3
    th = torch.from_numpy(random_theta(np.random.default_rng(5), n).astype(np.float32))
    comp, cost = (x.clone() for x in e.evaluate(th))
    for k in (1, 3, 4 * sms // per, 12 * sms // per, 12 * sms // per + 1, 16 * sms // per + 1, 24 * sms // per + 1):
        c, v = e.evaluate(th[5:5 + k])
        assert torch.equal(c, comp[5:5 + k]) and torch.equal(v, cost[5:5 + k]), k
