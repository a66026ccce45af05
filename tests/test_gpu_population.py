"""The lane layout's two families of rollout kernels against the FP64 oracle, each over its variants and motor shapes:
the population's (what a CEM and the server launch, one compiled copy for both) and, past the sizes that go to
four lanes a rollout, the evaluation's one-lane form. Tolerances as the layouts' parity tests: 1e-4 of the
oracle's cost scale."""
import numpy as np
import pytest
import torch

from helpers import oracle_windows, random_theta
from oracle import cost as oc
from oracle import dynamics as dyn
from oracle import go2_model as gm
from test_gpu_layouts import cost_error

pytestmark = pytest.mark.gpu
MOTORS = (dict(), dict(tanh_a=(15.0, 18.0, 25.0), motor_gain=(0.9, 1.1, 1.05), hip_action_scale=0.5))


def _case(kw, seed, N, W, H):
    sim = gm.SimParams(**{k: (np.asarray(v, dtype=np.float64) if isinstance(v, tuple) else v) for k, v in kw.items()})
    _, init, actions, target = oracle_windows(seed, n_traj=2, T=W + H, H=H, sim=sim)
    init, actions, target = init[:W], actions[:W], target[:W]
    th = random_theta(np.random.default_rng(seed), N).astype(np.float32)
    ref = dyn.rollout(np.tile(init.astype(np.float64), (N, 1)), np.tile(actions.astype(np.float64), (N, 1, 1)),
                      np.repeat(th.astype(np.float64), W, 0), sim)
    comp = oc.window_components(ref, np.tile(target.astype(np.float64), (N, 1))).reshape(N, W, 9)
    return [torch.from_numpy(a) for a in (init, actions, target)], torch.from_numpy(th), comp


@pytest.mark.parametrize("kw", MOTORS)
@pytest.mark.parametrize("W", [1, 37])
def test_population_kernels_match_oracle(built, kw, W):
    """The lane variants of a CEM's population on prior samples, plain and with window weights and the norm cost."""
    from spi_gb300.autotune import set_variant
    from spi_gb300.engine import COST_REF, COST_SQ, Engine
    from spi_gb300.robot import SimConfig
    windows, th, ref = _case(kw, 70 + W, 24, W, 10)
    e = Engine(SimConfig(**kw))
    weight = (np.arange(W) % 3 != 1).astype(np.float32)
    for w, norm, mode in ((None, None, COST_SQ), (weight, float(weight.sum()), COST_REF)):
        e.load_windows(*windows, None if w is None else torch.from_numpy(w), norm)
        e.set_cost(mode)
        mean = ref.mean(1) if w is None else (ref * w[None, :, None]).sum(1) / norm
        cost = oc.scalar_cost(mean) if mode == COST_SQ else oc.compute_cost(mean[:, :3])
        for variant in ("lane2", "lane3", "lane4"):
            set_variant(e, variant)
            e.set_theta(th)
            e.run(population=True)
            c, v = (x.cpu().numpy() for x in e.read())
            assert cost_error(c, mean) <= 1e-4 and cost_error(v, cost) <= 1e-4, variant
    assert e.sync() == 0


@pytest.mark.parametrize("kw", MOTORS)
def test_one_lane_evaluation_matches_oracle(built, kw):
    """2,000 (theta, group) pairs: between the 12 and the 16 an SM of 152 that go to the one-lane form."""
    from spi_gb300.autotune import set_variant
    from spi_gb300.engine import Engine
    from spi_gb300.robot import SimConfig
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert 12 * sms < 2000 <= 16 * sms
    windows, th, ref = _case(kw, 90, 200, 73, 3)
    e = Engine(SimConfig(**kw))
    e.load_windows(*windows)
    for variant in ("lane2", "lane3", "lane4"):
        set_variant(e, variant)
        c, v = (x.cpu().numpy() for x in e.evaluate(th))
        assert cost_error(c, ref.mean(1)) <= 1e-4 and cost_error(v, oc.scalar_cost(ref.mean(1))) <= 1e-4, variant
    assert e.sync() == 0
