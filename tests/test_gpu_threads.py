"""Engines used side by side on threads of one process."""
import threading

import numpy as np
import pytest
import torch

from helpers import oracle_windows, random_theta

pytestmark = pytest.mark.gpu


def test_sensitivities_of_two_engines_on_two_threads(built):
    """Five and thirteen directions, whose tangent kernels ask for different amounts of shared memory, in tight loops
    of library calls: every call succeeds, and each engine's last result is its first to the bit."""
    import ctypes

    from spi_gb300.engine import Engine
    from spi_gb300.robot import SimConfig
    from spi_gb300.sensitivity import sensitivities
    _, init, actions, target = oracle_windows(50, n_traj=2, T=160, H=1)
    windows = [torch.from_numpy(a[:257]) for a in (init, actions, target)]
    jobs = []
    for N, ids in ((20, (0, 3, 7, 8, 12)), (8, tuple(range(13)))):
        e = Engine(SimConfig(decimation=1), stream=torch.cuda.Stream())
        e.load_windows(*windows)
        th = torch.from_numpy(random_theta(np.random.default_rng(N), N).astype(np.float32)).cuda()
        torch.cuda.synchronize()
        with torch.cuda.stream(e.stream):
            first = sensitivities(e, th, ids)[0]
            jobs.append((e, th, ids, first, torch.zeros_like(first)))
    torch.cuda.synchronize()
    failures, gate = [], threading.Barrier(2)

    def work(e, th, ids, first, J):
        cids = (ctypes.c_int32 * len(ids))(*ids)
        call = lambda: e.lib.spi_sensitivity(e._h, th.data_ptr(), th.shape[0], cids, len(ids), J.data_ptr(), None)  # noqa: E731
        gate.wait(60)
        for _ in range(100):
            failures.extend((len(ids), rc) for rc in [call() for _ in range(100)] if rc)
            e.stream.synchronize()
        if not torch.equal(J, first):
            failures.append((len(ids), "differs"))
    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join(200)
    assert not any(t.is_alive() for t in threads)
    assert not failures, (len(failures), failures[:5])


def test_sensitivities_of_one_engine_on_two_streams(built):
    """An engine moved from one stream to another between calls, nothing waiting in between: the calls' results
    are those of each call alone, to the bit."""
    import ctypes

    from spi_gb300.engine import Engine
    from spi_gb300.sensitivity import sensitivities
    _, init, actions, target = oracle_windows(51, n_traj=2, T=160, H=5)
    e = Engine()
    e.load_windows(*(torch.from_numpy(a[:257]) for a in (init, actions, target)))
    thetas = [torch.from_numpy(random_theta(np.random.default_rng(s), 8).astype(np.float32)).cuda() for s in (1, 2)]
    alone = []
    for th in thetas:
        alone.append(sensitivities(e, th, range(13))[0])
        torch.cuda.synchronize()
    streams, ids = [torch.cuda.Stream() for _ in thetas], (ctypes.c_int32 * 13)(*range(13))
    outs = [[torch.zeros_like(alone[0]) for _ in range(10)] for _ in thetas]
    torch.cuda.synchronize()
    for i in range(10):
        for th, s, out in zip(thetas, streams, outs):
            assert e.lib.spi_set_stream(e._h, ctypes.c_void_p(s.cuda_stream)) == 0
            assert e.lib.spi_sensitivity(e._h, th.data_ptr(), 8, ids, 13, out[i].data_ptr(), None) == 0
    torch.cuda.synchronize()
    e.lib.spi_set_stream(e._h, ctypes.c_void_p(e.stream.cuda_stream))
    for out, ref in zip(outs, alone):
        assert all(torch.equal(o, ref) for o in out)
