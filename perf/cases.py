"""The work a user of this framework has it do, as cases that can be timed and compared.

Every case goes through a public entry point: batched candidate evaluation (``Engine.evaluate``),
a CEM identification, the continuous-batching server, the cost's gradient (``WindowCost``), state
sensitivities and Fisher information, the finite-difference Fisher objective, simulator stepping
and trajectory traces. Sizes come from the repository's own workloads (the one-parameter and the
13-parameter identification, the 20-point mass landscape, the served small-job mix, the scoring of
512 excitations) and from odd, ragged ones in between; ``draw`` gives more of the same ranges.

Inputs are made from the seed by a 64-bit simulation of the Go2 in plain torch (class ``Go2``
below), which also gives ``exact``: nothing in it uses the framework.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch
import torch.autograd.forward_ad as fwd

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "spi-active_gb300"))

from spi_gb300.active import fd_fisher  # noqa: E402
from spi_gb300.cem import CEM  # noqa: E402
from spi_gb300.engine import COST_REF, COST_SQ, DEFAULT_SQ_WEIGHTS, Engine  # noqa: E402
from spi_gb300.robot import SimConfig  # noqa: E402
from spi_gb300.sensitivity import WindowCost, fisher, sensitivities  # noqa: E402
from spi_gb300.server import Server, cem_config  # noqa: E402
from spi_gb300.sim import EngineSimulator  # noqa: E402

F64 = torch.float64
DEVICE = "cuda"

# theta: base mass, CoM offset 3, inertia scale, then Kp scale / friction / armature / torque-limit
# scale of the front and of the rear legs; the priors of the 13-parameter identification
NOMINAL = (6.921, 0.0, 0.0, 0.0, 1.0, 1.0, 0.0, 0.0, 1.0, 1.0, 0.0, 0.0, 1.0)
PRIOR_LO = (5.0, -0.05, -0.05, -0.05, 0.7, 0.8, 0.0, 0.0, 0.8, 0.8, 0.0, 0.0, 0.8)
PRIOR_HI = (9.0, 0.05, 0.05, 0.05, 1.3, 1.2, 0.3, 0.02, 1.0, 1.2, 0.3, 0.02, 1.0)
# the robot after half a second of standing with zero actions
STANDING = (0.0, 0.0, 0.26398, 0.0, -0.00662, 0.0, 0.99998, -0.08525, 0.0, 0.01163, 0.0, -0.11839, 0.0,
            0.22849, 0.68502, -1.71248, -0.22846, 0.68503, -1.7125, 0.20725, 1.0096, -1.78042, -0.20723, 1.0096,
            -1.78044, -0.03824, -0.23604, 0.25902, 0.03803, -0.23602, 0.25919, 0.16535, -0.19532, 0.02874,
            -0.16534, -0.19524, 0.02875)
CONTROL_DT = 0.005
ACTION_SCALE = 0.25
# FP operations of one rollout control step (four substeps of the condensed floating-base dynamics)
STEP_FLOPS = 20600


# ---------------------------------------------------------------------------------------------
# the Go2 in 64 bits
# ---------------------------------------------------------------------------------------------
def _t(x):
    return torch.tensor(x, dtype=F64, device=DEVICE)


def _sym(xx, yy, zz, xy, xz, yz):
    return [[xx, xy, xz], [xy, yy, yz], [xz, yz, zz]]


def _skew(a):
    z = torch.zeros_like(a[..., 0])
    return torch.stack([z, -a[..., 2], a[..., 1], a[..., 2], z, -a[..., 0], -a[..., 1], a[..., 0], z],
                       -1).reshape(*a.shape[:-1], 3, 3)


def _mv(A, x):
    return (A @ x[..., None])[..., 0]


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _inertia(m, c, about_com):
    """6x6 spatial inertia (angular first) of mass m at c with rotational inertia about its centre."""
    C = _skew(c)
    mC = m[..., None, None] * C
    eye = torch.eye(3, dtype=F64, device=DEVICE) * m[..., None, None]
    top = torch.cat([about_com - mC @ C, mC], -1)
    return torch.cat([top, torch.cat([-mC, eye.expand(mC.shape)], -1)], -2)


def _point(m, r):
    return _inertia(m, r, torch.zeros((*r.shape, 3), dtype=F64, device=DEVICE))


def _crm(v, m):
    """Spatial cross product v x m of motion vectors."""
    return torch.cat([_cross(v[..., :3], m[..., :3]), _cross(v[..., 3:], m[..., :3]) + _cross(v[..., :3], m[..., 3:])], -1)


def _crf(v, f):
    """Spatial cross product v x* f of a motion and a force vector."""
    return torch.cat([_cross(v[..., :3], f[..., :3]) + _cross(v[..., 3:], f[..., 3:]), _cross(v[..., :3], f[..., 3:])], -1)


def _rotation(q):
    x, y, z, w = q.unbind(-1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                        2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                        2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], -1).reshape(-1, 3, 3)


class Go2:
    """The floating-base dynamics of the engine in 64 bits: joint-space equations of the four legs
    and the base in base coordinates, penalty contacts with linearly implicit damping, PD and motor
    model, semi-implicit Euler. Differentiable in theta (forward mode)."""

    dt, substeps, g = 0.00125, 4, 9.81
    k, c, ct, mu, ramp = 2.0e4, 200.0, 200.0, 0.8, 1e-3
    kp, kd, friction_vel = 20.0, 0.5, 0.2

    def __init__(self, speed_limit=True):
        self.speed_limit = speed_limit
        mass, com, inertia, origin = [], [], [], []
        foot, foot_m = np.array([0.0, 0.0, -0.213]), 0.04
        for sx, sy in ((1, 1), (1, -1), (-1, 1), (-1, -1)):
            calf_m, calf_c = 0.154, np.array([0.00548, -0.000975 * sy, -0.115])
            m = calf_m + foot_m
            cc = (calf_m * calf_c + foot_m * foot) / m
            I = np.zeros((3, 3))
            for mm, p, J in ((calf_m, calf_c, np.array(_sym(0.00108, 0.0011, 3.29e-05, 3.4e-07 * sy, 1.72e-05, 8.28e-06 * sy))),
                             (foot_m, foot, 9.6e-6 * np.eye(3))):
                d = p - cc
                I += J + mm * (d @ d * np.eye(3) - np.outer(d, d))
            mass.append([0.678, 1.152, m])
            com.append([[-0.0054 * sx, 0.00194 * sy, -0.000105], [-0.00374, -0.0223 * sy, -0.0327], cc.tolist()])
            inertia.append([_sym(0.00048, 0.000884, 0.000596, -3.01e-06 * sx * sy, 1.11e-06 * sx, -1.42e-06 * sy),
                            _sym(0.00584, 0.0058, 0.00103, 8.72e-05 * sy, -0.000289, 0.000808 * sy), I.tolist()])
            origin.append([[0.1934 * sx, 0.0465 * sy, 0.0], [0.0, 0.0955 * sy, 0.0], [0.0, 0.0, -0.213]])
        self.mass, self.com, self.inertia, self.origin = _t(mass), _t(com), _t(inertia), _t(origin)
        self.foot = _t(foot.tolist())
        self.base_com, self.base_I = _t([0.021112, 0.0, -0.005366]), _t(_sym(0.02448, 0.098077, 0.107, 0.00012166, 0.0014849, -3.12e-05))
        heads = [_inertia(_t(0.001), _t(p), 9.6e-6 * torch.eye(3, dtype=F64, device=DEVICE)) for p in ([0.285, 0.0, 0.01], [0.293, 0.0, -0.06])]
        self.heads = heads[0] + heads[1]
        half = np.array([0.3762, 0.0935, 0.114]) / 2
        self.corners = _t([(half * np.array(s)).tolist() for s in ((a, b, c) for a in (1, -1) for b in (1, -1) for c in (1, -1))])
        self.q0 = _t([[0.1, 0.8, -1.5], [-0.1, 0.8, -1.5], [0.1, 1.0, -1.5], [-0.1, 1.0, -1.5]])
        self.tau_lim, self.vel_lim = _t([23.7, 23.7, 35.55]), _t([30.1, 30.1, 20.07])

    def _contact(self, pen, v):
        """World force on contact points at penetration pen with velocity v, and their implicit mass."""
        s = torch.clamp(pen / self.ramp, 0.0, 1.0)
        fn = torch.where(pen > 0, torch.relu(self.k * pen - self.c * s * v[..., 2]), torch.zeros_like(pen))
        vt2 = v[..., 0] ** 2 + v[..., 1] ** 2
        vt = torch.sqrt(torch.where(vt2 > 0, vt2, torch.ones_like(vt2)))
        lim = self.mu * fn
        scale = torch.where(self.ct * vt <= lim, torch.full_like(vt, self.ct), lim / vt)
        return torch.stack([-scale * v[..., 0], -scale * v[..., 1], fn], -1), self.dt * max(self.c, self.ct) * s

    def _motor(self, q, qd, target, th):
        leg = torch.stack([th[:, 5:9], th[:, 5:9], th[:, 9:13], th[:, 9:13]], 1)[..., None]   # [B, 4, 4, 1]
        tau = leg[:, :, 0] * self.kp * (target - q) - self.kd * qd
        lim = leg[:, :, 3] * self.tau_lim
        if self.speed_limit:
            lim = lim * torch.relu(1 - qd.abs() / self.vel_lim)
        lim = lim.expand_as(tau)
        tau = torch.minimum(torch.maximum(tau, -lim), lim)
        return tau - leg[:, :, 1] * torch.tanh(qd / self.friction_vel), leg[:, :, 2, 0]

    def _substep(self, st, target, th, Ib):
        p, quat, nu, q, qd = st
        R = _rotation(quat)
        up = R[:, 2, :]                                            # world vertical in base coordinates
        s0, c0 = torch.sin(q[..., 0]), torch.cos(q[..., 0])
        z, o = torch.zeros_like(s0), torch.ones_like(s0)

        def about_y(a):
            s, c = torch.sin(a), torch.cos(a)
            return torch.stack([c, z, s, z, o, z, -s, z, c], -1).reshape(*a.shape, 3, 3)
        Rh = torch.stack([o, z, z, z, c0, -s0, z, s0, c0], -1).reshape(*s0.shape, 3, 3)
        rot = [Rh, Rh @ about_y(q[..., 1]), Rh @ about_y(q[..., 1] + q[..., 2])]
        o0 = self.origin[:, 0].expand(*s0.shape, 3)
        o1 = o0 + _mv(rot[0], self.origin[:, 1])
        o2 = o1 + _mv(rot[1], self.origin[:, 2])
        foot = o2 + _mv(rot[2], self.foot)
        ax = torch.stack([o, z, z], -1)
        ay = Rh[..., 1]
        S = [torch.cat([a, _cross(r, a)], -1) for a, r in ((ax, o0), (ay, o1), (ay, o2))]
        V, A, v, a = [], [], nu[:, None].expand(-1, 4, -1), torch.zeros_like(S[0])
        for j in range(3):
            vj = S[j] * qd[..., j, None]
            v = v + vj
            a = a + _crm(v, vj)
            V.append(v)
            A.append(a)
        # foot contacts
        Rb = R[:, None]
        height = p[:, None, 2] + (up[:, None] * foot).sum(-1)
        vf = _mv(Rb, V[2][..., 3:] + _cross(V[2][..., :3], foot))
        F, mi = self._contact(0.022 - height, vf)
        F = _mv(Rb.transpose(-1, -2), F + torch.stack([z, z, mi * self.g], -1))
        # bodies
        I, f = [], []
        for j in range(3):
            Ij = _inertia(self.mass[:, j].expand_as(s0), (o0, o1, o2)[j] + _mv(rot[j], self.com[:, j]),
                          rot[j] @ self.inertia[:, j] @ rot[j].transpose(-1, -2))
            fj = _crf(V[j], _mv(Ij, V[j]))
            if j == 2:
                Ij = Ij + _point(mi, foot)
                fj = fj - torch.cat([_cross(foot, F), F], -1)
            I.append(Ij)
            f.append(fj + _mv(Ij, A[j]))
        for j in (1, 0):
            I[j] = I[j] + I[j + 1]
            f[j] = f[j] + f[j + 1]
        tau, arm = self._motor(q, qd, target, th)
        cols = [_mv(I[j], S[j]) for j in range(3)]
        M = torch.stack([torch.stack([(S[min(i, j)] * cols[max(i, j)]).sum(-1) for j in range(3)], -1) for i in range(3)], -2)
        M = M + torch.diag_embed(arm[..., None].expand(*arm.shape, 3))
        Fc = torch.stack(cols, -1)                                 # [B, 4, 6, 3]
        C = torch.stack([(S[j] * f[j]).sum(-1) for j in range(3)], -1)
        X = torch.linalg.solve(M, torch.cat([Fc.transpose(-1, -2), (tau - C)[..., None]], -1))
        # base: its own terms, the box corners, the legs
        H = Ib + (I[0] - Fc @ X[..., :6]).sum(1)
        b = _crf(nu, _mv(Ib, nu)) + (f[0] + _mv(Fc, X[..., 6])).sum(1)
        vc = _mv(Rb, nu[:, None, 3:] + _cross(nu[:, None, :3].expand(-1, 8, -1), self.corners.expand(p.shape[0], 8, 3)))
        Fk, mk = self._contact(-(p[:, None, 2] + up @ self.corners.T), vc)
        zk = torch.zeros_like(mk)
        Fk = _mv(Rb.transpose(-1, -2), Fk + torch.stack([zk, zk, mk * self.g], -1))
        cor = self.corners.expand(p.shape[0], 8, 3)
        H = H + _point(mk, cor).sum(1)
        b = b - torch.cat([_cross(cor, Fk), Fk], -1).sum(1)
        a0 = torch.linalg.solve(H, -b[..., None])[..., 0]
        qdd = X[..., 6] - (X[..., :6] @ a0[:, None, :, None])[..., 0]
        # integrate
        nu = nu + self.dt * (a0 - self.g * torch.cat([torch.zeros_like(up), up], -1))
        qd = qd + self.dt * qdd
        w = nu[:, :3]
        dq = torch.cat([quat[:, 3:] * w + _cross(quat[:, :3], w), -(w * quat[:, :3]).sum(-1, keepdim=True)], -1)
        quat = quat + 0.5 * self.dt * dq
        quat = quat / torch.sqrt((quat * quat).sum(-1, keepdim=True))
        p = p + self.dt * _mv(_rotation(quat), nu[:, 3:])
        return p, quat, nu, q + self.dt * qd, qd

    def rollout(self, x0, actions, theta, trace=False):
        """States after the last (or every) control step; x0 [B, 37], actions [B, H, 12], theta [B, 13]."""
        x0, actions, th = x0.to(F64), actions.to(F64), theta.to(F64)
        com = self.base_com + th[:, 1:4]
        scale = torch.ones_like(self.base_I) + torch.eye(3, dtype=F64, device=DEVICE) * (th[:, 4, None, None] - 1)
        Ib = _inertia(th[:, 0], com, self.base_I * scale) + self.heads
        R = _rotation(x0[:, 3:7])
        nu = torch.cat([_mv(R.transpose(-1, -2), x0[:, 10:13]), _mv(R.transpose(-1, -2), x0[:, 7:10])], -1)
        st = (x0[:, 0:3], x0[:, 3:7], nu, x0[:, 13:25].reshape(-1, 4, 3), x0[:, 25:37].reshape(-1, 4, 3))
        out = []
        for h in range(actions.shape[1]):
            target = torch.clamp(actions[:, h], -20.0, 20.0).reshape(-1, 4, 3) * ACTION_SCALE + self.q0
            for _ in range(self.substeps):
                st = self._substep(st, target, th, Ib)
            if trace or h == actions.shape[1] - 1:
                p, quat, nu, q, qd = st
                R = _rotation(quat)
                out.append(torch.cat([p, quat, _mv(R, nu[:, 3:]), _mv(R, nu[:, :3]), q.flatten(1), qd.flatten(1)], -1))
        return torch.stack(out, 1) if trace else out[-1]

    def tangents(self, x0, actions, theta, direction):
        """Final states and their derivative along direction [B, 13] in theta."""
        with fwd.dual_level(), torch.no_grad():
            p = fwd.unpack_dual(self.rollout(x0, actions, fwd.make_dual(theta.to(F64), direction.to(F64))))
            return p.primal, p.tangent


# ---------------------------------------------------------------------------------------------
# inputs from the seed
# ---------------------------------------------------------------------------------------------
def _rng(seed, salt):
    return np.random.default_rng([int(seed), salt])


def _dev(a):
    return torch.as_tensor(np.asarray(a, np.float32), device=DEVICE)


def _thetas(rng, n, dims=13):
    """Samples of the prior; the slots past the first dims at their nominal value."""
    th = np.tile(np.array(NOMINAL), (n, 1))
    lo, hi = np.array(PRIOR_LO), np.array(PRIOR_HI)
    th[:, :dims] = lo[:dims] + (hi - lo)[:dims] * rng.random((n, dims))
    return th


def _sines(rng, n, T, amp=(0.1, 0.4), freq=(1.0, 3.0), parts=1):
    """Raw actions [n, T, 12]: per joint a sum of sines of joint target."""
    a, f = rng.uniform(*amp, (n, 12, parts)) / math.sqrt(parts), rng.uniform(*freq, (n, 12, parts))
    ph = rng.uniform(0.0, 2 * np.pi, (n, 12, parts))
    t = np.arange(T)[:, None, None] * CONTROL_DT
    return (a[:, None] * np.sin(2 * np.pi * f[:, None] * t + ph[:, None])).sum(-1).astype(np.float32) / ACTION_SCALE


def _stand(rng, n):
    """Standing robots, each a little off in pose and velocity."""
    x = np.tile(np.array(STANDING), (n, 1))
    x[:, 7:13] += 0.05 * rng.standard_normal((n, 6))
    x[:, 13:25] += 0.02 * rng.standard_normal((n, 12))
    x[:, 25:37] += 0.2 * rng.standard_normal((n, 12))
    return x


def _windows(seed, W, H, speed_limit=True):
    """W logged windows of H control steps of robots under sine excitation: init [W, 37], actions
    [W, H, 12], target [W, 37] (the state the true parameters reach), and the true parameters."""
    rng = _rng(seed, 1)
    lead = 12
    true = _thetas(rng, 1)
    acts = _dev(_sines(rng, W, lead + H))
    th = _t(true).expand(W, 13)
    sim = Go2(speed_limit)
    with torch.no_grad():
        init = sim.rollout(_t(_stand(rng, W)), acts[:, :lead], th).float()
        target = sim.rollout(init, acts[:, lead:].contiguous(), th).float()
    return init, acts[:, lead:].contiguous(), target


def _job_windows(seed, sizes):
    """The windows of several jobs (each with its own true parameters), from one simulation."""
    rng = _rng(seed, 2)
    lead, longest, n = 12, max(H for _, _, H, _ in sizes), sum(W for _, W, _, _ in sizes)
    acts = _dev(_sines(rng, n, lead + longest))
    th = _t(np.repeat(_thetas(rng, len(sizes)), [W for _, W, _, _ in sizes], 0))
    sim = Go2()
    with torch.no_grad():
        init = sim.rollout(_t(_stand(rng, n)), acts[:, :lead], th).float()
        states = sim.rollout(init, acts[:, lead:], th, trace=True).float()
    at, out = 0, []
    for _, W, H, _ in sizes:
        rows = slice(at, at + W)
        out.append((init[rows].contiguous(), acts[rows, lead:lead + H].contiguous(), states[rows, H - 1].contiguous()))
        at += W
    return out


def _config(case):
    return SimConfig() if case.get("speed_limit", True) else SimConfig.reference_compatible()


def _prior(dims):
    return np.array(PRIOR_LO[:dims]), np.array(PRIOR_HI[:dims])


def _job_sizes(case):
    """Sizes of the served jobs, log-uniform over the small-job ranges."""
    rng = np.random.default_rng(case["mix"])

    def u(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return [(u(64, case["pop"]), u(8, case["windows"]), u(5, case["H"]), int(rng.integers(1, 14))) for _ in range(case["jobs"])]


# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------
def listed():
    return [
        # one step of the one-parameter (base mass) identification: the smallest call, all latency
        dict(name="eval_mass64", kind="eval", N=64, W=8, H=5, dims=1, speed_limit=True, cost="sq"),
        # the 20-point mass landscape of a logged file: the reference's cost, torque path and window mask
        dict(name="eval_landscape", kind="eval", N=20, W=195, H=5, dims=1, speed_limit=False, cost="ref"),
        # an ordinary batch of odd sizes
        dict(name="eval_odd", kind="eval", N=333, W=37, H=11, dims=13, speed_limit=True, cost="sq"),
        # one iteration's evaluation of the full 13-parameter identification: the largest call
        dict(name="eval_full", kind="eval", N=4096, W=256, H=20, dims=13, speed_limit=True, cost="sq"),
        # a small identification job from its start to its result
        dict(name="cem_job", kind="cem", N=512, W=64, H=20, dims=5, iterations=2),
        # small jobs of uneven sizes through the continuous-batching server
        dict(name="serve_small", kind="serve", jobs=24, pop=512, windows=64, H=20, iterations=2, mix=1),
        # cost and gradient of a population, as a gradient-based identification calls them
        dict(name="grad_full", kind="grad", N=512, W=256, H=20),
        # 13 state sensitivities of the windows of 512 candidate excitations
        dict(name="sens_512x8", kind="sens", N=1, W=4096, H=20, K=13),
        # Fisher information and log det of those candidates on the tensor cores
        dict(name="fisher_512x8", kind="fisher", N=512, W=8, K=13, tensor_cores=True),
        # the finite-difference Fisher objective of a population of excitations (13 auxiliary robots each)
        dict(name="fd_512x13", kind="fd", C=512, T=200, P=13, ksync=5),
        # a vectorised simulator step
        dict(name="step_4096", kind="step", B=4096, steps=1),
        # trajectories of candidate excitations, every state kept
        dict(name="trace_512", kind="trace", W=512, T=180),
    ]


def draw(rng):
    def u(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["eval", "eval", "eval", "cem", "serve", "grad", "sens", "fisher", "fd", "step", "trace"])
    if kind == "eval":
        N, W, H = u(8, 4096), u(4, 512), u(5, 50)
        while N * W * H > 4096 * 256 * 20:
            N = N // 2
        return dict(kind=kind, N=N, W=W, H=H, dims=rng.choice([1, 5, 13]), speed_limit=rng.random() < 0.7,
                    cost=rng.choice(["sq", "sq", "ref"]))
    if kind == "cem":
        return dict(kind=kind, N=u(64, 1024), W=u(8, 256), H=rng.randint(5, 20), dims=rng.randint(1, 13), iterations=rng.randint(1, 2))
    if kind == "serve":
        return dict(kind=kind, jobs=rng.randint(4, 24), pop=u(128, 512), windows=u(16, 64), H=rng.randint(6, 20), iterations=2,
                    mix=rng.randint(2, 10 ** 6))
    if kind == "grad":
        N, W = u(4, 512), u(8, 256)
        return dict(kind=kind, N=N, W=W, H=rng.randint(5, 20))
    if kind == "sens":
        return dict(kind=kind, N=rng.randint(1, 3), W=u(16, 1365), H=rng.randint(5, 20), K=rng.randint(1, 13))
    if kind == "fisher":
        return dict(kind=kind, N=u(1, 1024), W=u(1, 64), K=rng.randint(1, 13), tensor_cores=rng.random() < 0.5)
    if kind == "fd":
        return dict(kind=kind, C=u(16, 512), T=u(50, 200), P=rng.randint(1, 13), ksync=rng.choice([1, 3, 5, 10]))
    if kind == "step":
        return dict(kind=kind, B=u(1, 8192), steps=rng.randint(1, 4))
    return dict(kind="trace", W=u(1, 512), T=u(25, 180))


def prepare(case, seed):
    kind = case["kind"]
    rng = _rng(seed, 0)
    s = dict(case=case)
    if kind in ("eval", "cem", "grad", "sens"):
        s["init"], s["actions"], s["target"] = _windows(seed, case["W"], case["H"], case.get("speed_limit", True))
        s["engine"] = e = Engine(_config(case))
        weight = norm = None
        if case.get("cost") == "ref":      # the reference masks the windows that run past a file's end
            weight = torch.ones(case["W"], device=DEVICE)
            weight[case["W"] - case["W"] // 8:] = 0.0
            norm = float(weight.sum())
        s["weight"], s["norm"] = weight, norm
        e.load_windows(s["init"], s["actions"], s["target"], weight, norm)
        e.set_cost(COST_REF if case.get("cost") == "ref" else COST_SQ, DEFAULT_SQ_WEIGHTS)
        if kind != "cem":
            s["theta"] = _dev(_thetas(rng, case["N"], case.get("dims", 13)))
    elif kind == "serve":
        s["server"] = srv = Server(max_slots=32, max_samples=512, hbm_budget_bytes=8 << 30)
        srv.set_variant("lane3")
        srv.set_rounds(4)
        sizes = _job_sizes(case)
        s["windows"], s["jobs"] = _job_windows(seed, sizes), []
        for j, (pop, W, H, dims) in enumerate(sizes):
            lo, hi = _prior(dims)
            cem = cem_config(pop, list(range(dims)), lo, hi, NOMINAL, seed=1000 + j, job_id=j)
            s["jobs"].append(Server.make_job(*s["windows"][j], cem, case["iterations"]))
    elif kind == "fisher":
        # Jacobians of the size the windows of an excitation give: each parameter has a scale of its own
        scale = np.array([0.02, 0.6, 0.9, 0.5, 0.03, 0.3, 0.07, 3.5, 0.01, 0.25, 0.07, 2.8, 0.01])[:case["K"]]
        gen = torch.Generator(device=DEVICE).manual_seed(int(seed))
        s["J"] = torch.randn((case["N"], case["W"], 37, case["K"]), device=DEVICE, generator=gen) * _dev(scale)
        s["weight"] = _dev(np.repeat(np.array(DEFAULT_SQ_WEIGHTS), (3, 4, 3, 3, 12, 12)))
    elif kind == "fd":
        s["engine"] = Engine()
        x = np.tile(np.array(STANDING), (case["C"], 1))
        s["init"] = _dev(x)
        s["actions"] = _dev(_sines(rng, case["C"], case["T"], amp=(0.05, 0.4), freq=(0.5, 4.0), parts=3))
        s["theta"] = _dev(_thetas(rng, 1)[0])
    elif kind == "step":
        s["sim"] = sim = EngineSimulator(case["B"])
        s["init"] = _dev(_stand(rng, case["B"]))
        sim.state.copy_(s["init"])
        s["theta"] = _dev(_thetas(rng, case["B"]))
        sim.set_theta(s["theta"])
        s["actions"] = _dev(rng.uniform(-0.8, 0.8, (case["B"], case["steps"], 12)))
    else:
        s["engine"] = e = Engine()
        s["init"] = _dev(_stand(rng, case["W"]))
        acts = _sines(rng, case["W"], case["T"], amp=(0.05, 0.4), freq=(0.5, 4.0), parts=3)
        acts[:, :case["T"] // 2] = 0.0       # the first half settles
        s["actions"] = _dev(acts)
        e.load_windows(s["init"], s["actions"], s["init"])
        s["theta"] = _dev(_thetas(rng, 1))
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "eval":
        comp, cost = s["engine"].evaluate(s["theta"])
        return {"comp": comp, "cost": cost}
    if kind == "cem":
        dims = case["dims"]
        lo, hi = _prior(dims)
        cem = CEM(s["engine"], case["N"], list(range(dims)), lo, hi, NOMINAL, seed=7)
        cem.run(case["iterations"])
        r = cem.read()
        return {"mu": r["mu"], "cov": r["cov"], "best_theta": r["best_theta"], "best_cost": r["best_cost"], "theta": cem.theta()}
    if kind == "serve":
        srv = s["server"]
        for j in s["jobs"]:
            srv.submit(j)
        done = srv.run_until_done(len(s["jobs"]))
        return {"best_cost": [done[j]["best_cost"] for j in sorted(done)],
                "best_theta": np.stack([done[j]["best_theta"] for j in sorted(done)]),
                "mu": np.concatenate([done[j]["mu"] for j in sorted(done)])}
    if kind == "grad":
        theta = s["theta"].clone().requires_grad_(True)
        cost = WindowCost.apply(theta, s["engine"], DEFAULT_SQ_WEIGHTS)
        cost.sum().backward()
        return {"cost": cost.detach(), "grad": theta.grad}
    if kind == "sens":
        J, x = sensitivities(s["engine"], s["theta"], range(case["K"]))
        return {"J": J, "x": x}
    if kind == "fisher":
        F, logdet, trace = fisher(s["J"], s["weight"], tensor_cores=case["tensor_cores"])
        return {"F": F, "logdet": logdet, "trace": trace}
    if kind == "fd":
        obj, rewards = fd_fisher(s["engine"], s["init"], s["actions"], s["theta"], list(range(case["P"])), ksync=case["ksync"], trace=True)
        return {"objective": obj, "rewards": rewards}
    if kind == "step":
        s["sim"].step(s["actions"], case["steps"])
        return {"state": s["sim"].state}
    comp, cost, trace = s["engine"].evaluate(s["theta"], trace=True)
    return {"comp": comp, "cost": cost, "trace": trace}


def work(case):
    """Bytes of the inputs and outputs, and the operations of the dynamics' recursive equations: a
    tangent direction costs about one more forward pass, the reverse sweep about two."""
    kind = case["kind"]
    window = lambda W, H: 4 * W * (2 * 37 + 12 * H + 1)  # noqa: E731
    if kind in ("eval", "grad"):
        N, W, H = case["N"], case["W"], case["H"]
        out = 10 if kind == "eval" else 14
        return {"bytes": window(W, H) + 4 * N * (13 + out), "flops": N * W * H * STEP_FLOPS * (1 if kind == "eval" else 4)}
    if kind == "cem":
        N, W, H = case["N"], case["W"], case["H"]
        return {"bytes": window(W, H) + 4 * N * 13, "flops": case["iterations"] * N * W * H * STEP_FLOPS}
    if kind == "serve":
        sizes = _job_sizes(case)
        return {"bytes": sum(window(W, H) + 4 * 13 * N for N, W, H, _ in sizes),
                "flops": case["iterations"] * STEP_FLOPS * sum(N * W * H for N, W, H, _ in sizes)}
    if kind == "sens":
        N, W, H, K = case["N"], case["W"], case["H"], case["K"]
        return {"bytes": window(W, H) + 4 * N * W * 37 * (K + 1), "flops": N * W * H * STEP_FLOPS * (1 + K)}
    if kind == "fisher":
        N, W, K = case["N"], case["W"], case["K"]
        return {"bytes": 4 * N * W * 37 * K + N * (4 * K * K + 16), "flops": N * W * 37 * K * (K + 2)}
    if kind == "fd":
        C, T, P = case["C"], case["T"], case["P"]
        return {"bytes": 4 * C * (37 + T * 13), "flops": C * (P + 1) * (T + 1) * STEP_FLOPS}
    if kind == "step":
        B, n = case["B"], case["steps"]
        return {"bytes": 4 * B * (2 * 37 + 13 + 12 * n), "flops": B * n * STEP_FLOPS}
    W, T = case["W"], case["T"]
    return {"bytes": 4 * W * (2 * 37 + 12 * T + 37 * T), "flops": W * T * STEP_FLOPS}


# ---------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------
def _components(x, target, weight, norm):
    """Weighted mean error components [N, 9] of final states [N, W, 37]."""
    d = x - target.to(F64)
    sq = [(b * b).sum(-1) for b in d.split((3, 4, 3, 3, 12, 12), -1)]
    comp = torch.stack([sq[0].sqrt(), sq[1].sqrt(), sq[4].sqrt()] + sq, -1)
    return (comp * weight[None, :, None]).sum(1) / norm


def _pairs(s, tangents=1):
    """Every (theta, window) pair (times the tangent directions) as one batch."""
    N, W = s["theta"].shape[0], s["init"].shape[0]
    n = N * W * tangents
    return (s["init"][None, :, None].expand(N, W, tangents, 37).reshape(n, 37),
            s["actions"][None, :, None].expand(N, W, tangents, -1, 12).reshape(n, -1, 12),
            s["theta"][:, None, None].expand(N, W, tangents, 13).reshape(n, 13))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("cem", "serve"):             # sampled populations: the generator is the framework's own
        return None
    steps = {"eval": lambda c: c["N"] * c["W"] * c["H"], "grad": lambda c: 13 * c["N"] * c["W"] * c["H"],
             "sens": lambda c: c["K"] * c["N"] * c["W"] * c["H"], "fd": lambda c: c["C"] * (c["P"] + 1) * c["T"]}
    if kind in steps and steps[kind](case) > 1_500_000:
        return None                          # more than 20 seconds
    s = prepare(case, seed)
    sim = Go2(case.get("speed_limit", True))
    sq = _t(DEFAULT_SQ_WEIGHTS)
    with torch.no_grad():
        if kind in ("eval", "trace"):
            W = s["init"].shape[0]
            weight = s["weight"].to(F64) if s.get("weight") is not None else torch.ones(W, dtype=F64, device=DEVICE)
            norm = s.get("norm") or W
            x = sim.rollout(*_pairs(s), trace=kind == "trace")
            last = x[:, -1] if kind == "trace" else x
            target = s["target"] if kind == "eval" else s["init"]
            comp = _components(last.reshape(-1, W, 37), target, weight, norm)
            cost = 10 * comp[:, 0] + 5 * comp[:, 1] + comp[:, 2] if case.get("cost") == "ref" else comp[:, 3:] @ sq
            out = {"comp": comp, "cost": cost}
            if kind == "trace":
                out["trace"] = x[None]
            return out
        if kind in ("grad", "sens"):
            K = 13 if kind == "grad" else case["K"]
            x0, acts, th = _pairs(s, K)
            direction = torch.eye(13, dtype=F64, device=DEVICE)[:K].repeat(x0.shape[0] // K, 1)
            x, d = sim.tangents(x0, acts, th, direction)
            x, d = (v.reshape(s["theta"].shape[0], -1, K, 37) for v in (x, d))
            if kind == "sens":
                return {"J": d.transpose(-1, -2), "x": x[:, :, 0]}
            q = torch.repeat_interleave(sq, _t([3, 4, 3, 3, 12, 12]).long())
            diff = x[:, :, 0] - s["target"].to(F64)
            return {"cost": (q * diff * diff).sum(-1).mean(1), "grad": 2 * torch.einsum("nwi,i,nwki->nk", diff, q, d) / s["init"].shape[0]}
        if kind == "fisher":
            J, q = s["J"].to(F64), s["weight"].to(F64)
            F = torch.einsum("nwik,i,nwil->nkl", J, q, J)
            return {"F": F, "logdet": torch.logdet(F + 1e-9 * torch.eye(case["K"], dtype=F64, device=DEVICE)),
                    "trace": torch.diagonal(F, dim1=1, dim2=2).sum(-1)}
        if kind == "step":
            return {"state": sim.rollout(s["init"], s["actions"], s["theta"])}
        # fd: the main robot and one auxiliary per parameter, which take the main's state after the
        # zero-action reset step and then every ksync steps (every step for ksync = 1)
        C, P, ksync = case["C"], case["P"], case["ksync"]
        G = P + 1
        th = s["theta"].to(F64)[None, None].repeat(C, G, 1)
        for k in range(P):
            th[:, k + 1, k] += 0.1
        th = th.reshape(C * G, 13)
        x = s["init"].to(F64)[:, None].expand(C, G, 37).reshape(C * G, 37)
        acts = torch.cat([torch.zeros((C, 1, 12), dtype=F64, device=DEVICE), s["actions"].to(F64)], 1)
        rewards = []
        for t in range(acts.shape[1]):
            x = sim.rollout(x, acts[:, None, t:t + 1].expand(C, G, 1, 12).reshape(C * G, 1, 12), th)
            y = x.reshape(C, G, 37)
            d = (y[:, :1, :25] - y[:, 1:, :25]) / 0.1
            rewards.append((d * d).sum((1, 2)))
            if ksync <= 1 or (t + 1) % ksync == 1:
                x = y[:, :1].expand(C, G, 37).reshape(C * G, 37)
        rewards = torch.stack(rewards[1:], 1)
        return {"objective": rewards.sum(1) / (case["T"] + 1), "rewards": rewards}
