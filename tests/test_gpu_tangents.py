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
