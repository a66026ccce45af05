"""Sensitivities of many pairs: direction 0 as a dual rollout that keeps its substeps, the others by tangents
from them, against the dual rollouts that few pairs take."""
import numpy as np
import pytest
import torch

from helpers import oracle_windows, random_theta

pytestmark = pytest.mark.gpu


# 257 windows a theta; three to thirteen directions, counts that do and do not divide a CTA's 32
# quads; the first line's pairs are more than 4 GB of kept substeps hold, the last three's share
# their tapes
@pytest.mark.parametrize("N,ids", [(281, (0, 11, 5)), (16, (0, 3, 7, 8, 12)), (10, (1, 2, 4, 5, 6, 9, 10, 12)),
                                   (6, tuple(range(13))), (20, (0, 3, 7, 8, 12)), (12, (1, 2, 4, 5, 6, 9, 10, 12)),
                                   (8, tuple(range(13)))])
def test_tangents_agree_with_dual_rollouts(built, N, ids):
    """Final states to the bit, J within the 1e-3 that it is held to everywhere; a second call to the bit."""
    from spi_gb300.engine import Engine
    from spi_gb300.sensitivity import sensitivities
    _, init, actions, target = oracle_windows(33, n_traj=2, T=160, H=20)
    init, actions, target = (torch.from_numpy(a[:257]) for a in (init, actions, target))
    assert init.shape[0] == 257
    e = Engine()
    e.load_windows(init, actions, target)
    th = torch.from_numpy(random_theta(np.random.default_rng(5), N).astype(np.float32))
    J, x = sensitivities(e, th, list(ids))
    J2, x2 = sensitivities(e, th, list(ids))
    assert torch.equal(J, J2) and torch.equal(x, x2)
    for n in (0, N // 2, N - 1):
        ref, rx = sensitivities(e, th[n:n + 1], list(ids))
        assert torch.equal(x[n], rx[0])
        assert torch.linalg.norm(J[n] - ref[0]) <= 1e-3 * torch.linalg.norm(ref[0])


def _falling(rng):
    """Level bases a metre up with purely vertical velocities, powers of two, and resting joints: every foot
    off the ground, its sideways speed zero or a rounding."""
    from oracle import go2_model as gm
    x = np.zeros((257, 37), dtype=np.float32)
    x[:, 2], x[:, 6], x[:, 13:25] = 1.0, 1.0, gm.DEFAULT_DOF_POS
    x[:, 9] = rng.choice([-1.0, -0.5, -0.25, 0.125, 0.25, 0.5, 1.0], 257)
    return x


def _grounded(rng):
    """Bases lying on the ground on folded legs, some moving straight up or down: corners on and off."""
    x = np.zeros((257, 37), dtype=np.float32)
    x[:, 2], x[:, 6], x[:, 13:25] = 0.057 + rng.uniform(-1e-3, 2e-3, 257), 1.0, np.tile([0.0, 1.5, -3.0], 4)
    x[:, 9] = rng.choice([0.0, -0.25, 0.125, 0.25], 257)
    return x


@pytest.mark.parametrize("start,kw", [
    (None, dict()), (None, dict(torque_speed=False, inertia_follows_mass=True)),
    (None, dict(tanh_a=(15.0, 18.0, 25.0), motor_gain=(0.9, 1.1, 1.05))), (_falling, dict()), (_grounded, dict())])
def test_each_direction_agrees_with_its_dual_rollout(built, start, kw):
    """Column by column, since the directions' scales span a factor of 1e4: each within 1e-4 of its own norm over a
    theta's windows (some tens of FP32 roundings, amplified by the contacts' stiffness; 7e-6 was the largest of
    20 other input sets). A column that is zero, such as a torque limit never reached, is zero in both."""
    from oracle import go2_model as gm
    from spi_gb300.engine import Engine
    from spi_gb300.robot import SimConfig
    from spi_gb300.sensitivity import sensitivities
    rng = np.random.default_rng(40)
    if start is None:
        sim = gm.SimParams(**{k: (np.asarray(v, dtype=np.float64) if isinstance(v, tuple) else v) for k, v in kw.items()})
        _, init, actions, target = oracle_windows(41, n_traj=2, T=160, H=20, sim=sim)
        init, actions, target = init[:257], actions[:257], target[:257]
    else:
        init = target = start(rng)
        actions = rng.uniform(-1.0, 1.0, (257, 20, 12)).astype(np.float32)
        actions[:64] = 0.0
    e = Engine(SimConfig(**kw))
    e.load_windows(*(torch.from_numpy(np.ascontiguousarray(a)) for a in (init, actions, target)))
    th = torch.from_numpy(random_theta(rng, 7).astype(np.float32))
    J, x = sensitivities(e, th, list(range(13)))
    assert torch.isfinite(J).all()
    for n in range(7):
        ref, rx = sensitivities(e, th[n:n + 1], list(range(13)))
        assert torch.equal(x[n], rx[0])
        err, size = (torch.linalg.norm(a.reshape(-1, 13), dim=0) for a in (J[n] - ref[0], ref[0]))
        assert (err <= 1e-4 * size).all(), (n, err, size)


def test_little_memory_takes_smaller_batches(built):
    """70,000 windows keep 4.2 GB in one batch. With 3 GB left, every call succeeds and gives the bits that it gives
    with all of it (a window does not depend on its batch); with 0.1 GB left they are the dual rollouts'."""
    from spi_gb300.data import standing_state
    from spi_gb300.engine import Engine
    from spi_gb300.sensitivity import sensitivities
    gen = torch.Generator(device="cuda").manual_seed(1)
    init = torch.from_numpy(standing_state(70000)).cuda()
    actions = 1.2 * torch.rand((70000, 20, 12), device="cuda", generator=gen) - 0.6
    th = torch.from_numpy(random_theta(np.random.default_rng(2), 1).astype(np.float32))

    def run(left):
        e = Engine()
        e.load_windows(init, actions, init)
        hog = None
        torch.cuda.empty_cache()
        spare = torch.empty((2, 70000, 37, 13), device="cuda")     # the calls' results come from torch's cache
        del spare
        if left:
            hog = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
        outs = [sensitivities(e, th, range(13)) for _ in range(2)]
        torch.cuda.synchronize()
        del hog
        torch.cuda.empty_cache()                                   # back to the device, for what allocates outside torch
        e.close()
        assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
        return outs[0]
    J, x = run(None)
    J2, x2 = run(3 << 30)
    assert torch.equal(J, J2) and torch.equal(x, x2)
    del J2, x2
    J3, x3 = run(100 << 20)
    assert torch.equal(x, x3)
    assert (torch.linalg.norm((J - J3).reshape(-1, 13), dim=0) <= 1e-4 * torch.linalg.norm(J3.reshape(-1, 13), dim=0)).all()
