"""The kernel's dynamics source (csrc/dynamics.cuh), built for the host in FP64, against the oracle.

Proves on the CPU that the equations the sm_103a kernel executes are the oracle's
equations; the GPU tests then only have FP32 rounding and the lane plumbing to check.
"""
import ctypes

import numpy as np
import pytest

from oracle import dynamics as dyn
from oracle import go2_model as gm
from oracle import spatial
from oracle import sysid as osy
from helpers import random_theta

# Instrumented counts at the default configuration and a standing state (base-box corners off
# the ground): the articulated-body formulation of the oracle (csrc/aba_reference.h), the
# roofline's algorithmic figure, and the kernel's condensed formulation (csrc/dynamics.cuh; the
# joint targets of the actions are formed once per control step, outside the substep).
FLOPS_PER_SUBSTEP = 7053
EXECUTED_FLOPS_PER_SUBSTEP = 5149


def _emu(built, cfg, x0, acts, th):
    from spi_gb300 import _lib, robot
    r = robot.to_struct(cfg)
    B, H = acts.shape[:2]
    out = np.zeros((B, H, 37))
    x0c, ac, tc = (np.ascontiguousarray(a, dtype=np.float64) for a in (x0, acts, th))
    rc = _lib.hostemu_lib().spi_hostemu_rollout(ctypes.byref(r), x0c.ctypes.data, ac.ctypes.data,
                                                tc.ctypes.data, B, H, out.ctypes.data)
    assert rc == 0
    return out, r


@pytest.fixture
def oracle_f32_constants(monkeypatch):
    """Patch the oracle's constants to the float32 values the C struct carries."""
    from spi_gb300 import robot
    r = robot.to_struct(robot.SimConfig())
    org = np.zeros((13, 3))
    Irig = dyn._I_RIGID.copy()
    for b in range(12):
        h = np.array(r.body_h[b][:], dtype=np.float64)
        I6 = np.array(r.body_I[b][:], dtype=np.float64)
        M6 = np.zeros((6, 6))
        M6[:3, :3] = [[I6[0], I6[3], I6[4]], [I6[3], I6[1], I6[5]], [I6[4], I6[5], I6[2]]]
        M6[:3, 3:] = spatial.skew(h)
        M6[3:, :3] = spatial.skew(h).T
        M6[3:, 3:] = r.body_mass[b] * np.eye(3)
        Irig[b + 1] = M6
        org[b + 1] = np.array(r.body_origin[b][:], dtype=np.float64)
    fI = np.array(r.fixed_I[:], dtype=np.float64)
    fh = np.array(r.fixed_h[:], dtype=np.float64)
    H6 = np.zeros((6, 6))
    H6[:3, :3] = [[fI[0], fI[3], fI[4]], [fI[3], fI[1], fI[5]], [fI[4], fI[5], fI[2]]]
    H6[:3, 3:] = spatial.skew(fh)
    H6[3:, :3] = spatial.skew(fh).T
    H6[3:, 3:] = r.fixed_mass * np.eye(3)
    f = lambda a: np.asarray(a, dtype=np.float32).astype(np.float64)   # noqa: E731
    monkeypatch.setattr(dyn, "_ORIGIN", org)
    monkeypatch.setattr(dyn, "_I_RIGID", Irig)
    monkeypatch.setattr(dyn, "_I_HEADS", H6)
    for name in ("BASE_COM", "BASE_INERTIA", "FOOT_IN_CALF", "BASE_CORNERS"):
        monkeypatch.setattr(gm, name, f(getattr(gm, name)))
    return gm.SimParams(sim_dt=float(np.float32(0.00125)), gravity=float(np.float32(9.81)),
                        contact_mu=float(np.float32(0.8)), foot_radius=float(np.float32(0.022)),
                        friction_vel=float(np.float32(0.2)), torque_limit=f(gm.TORQUE_LIMIT),
                        contact_ramp=1.0 / float(np.float32(1.0) / np.float32(1e-3)),
                        velocity_limit=f(gm.VELOCITY_LIMIT), default_dof_pos=f(gm.DEFAULT_DOF_POS))


def _inputs(seed, B=12, H=8):
    from spi_gb300 import robot
    rng = np.random.default_rng(seed)
    cfg = robot.SimConfig()
    th = np.asarray(random_theta(rng, B), dtype=np.float32).astype(np.float64)
    x0 = osy.standing_state(B, z=0.30)
    x0[:, 7:13] = 0.3 * rng.normal(size=(B, 6))
    x0[:, 25:] = rng.normal(size=(B, 12))
    acts = osy.sine_actions(H, rng.uniform(0.1, 0.4, (B, 12)), rng.uniform(1, 3, (B, 12)),
                            rng.uniform(0, 6.28, (B, 12)), cfg.control_dt, cfg.action_scale)
    return cfg, x0, acts, th


def test_kernel_equations_equal_oracle(built, oracle_f32_constants):
    cfg, x0, acts, th = _inputs(11)
    emu, _ = _emu(built, cfg, x0, acts, th)
    ref = dyn.rollout(x0, acts, th, oracle_f32_constants, trace=True)
    assert np.abs(emu - ref).max() < 1e-9


def test_kernel_equations_reference_motor_variants(built, oracle_f32_constants):
    """Reference torque path (plain clip), tanh motor model and hip x0.5, contacts off/on."""
    from spi_gb300 import robot
    cfg, x0, acts, th = _inputs(12)
    for kw in (dict(torque_speed=False), dict(tanh_a=(15.0, 18.0, 25.0), hip_action_scale=0.5),
               dict(base_contact=False, motor_gain=(0.9, 1.1, 1.05))):
        c = robot.SimConfig(**kw)
        emu, _ = _emu(built, c, x0, acts, th)
        sp = oracle_f32_constants
        sp2 = gm.SimParams(**{**sp.__dict__, **{k: (np.asarray(v, dtype=np.float32).astype(np.float64) if isinstance(v, tuple) else v)
                                                 for k, v in kw.items()}})
        ref = dyn.rollout(x0, acts, th, sp2, trace=True)
        assert np.abs(emu - ref).max() < 1e-9, kw


def test_condensed_legs_equal_articulated_body_algorithm(built):
    """The kernel's leg condensation (joint-space inertia + Schur complement) and the oracle's
    articulated-body algorithm, both in FP64 with the same constants, agree to rounding, in
    and out of contact."""
    from spi_gb300 import _lib, robot
    cfg, x0, acts, th = _inputs(15, B=16, H=12)
    x0[:8, 2] = 0.26                                   # half the rollouts start with feet pressed in
    emu, r = _emu(built, cfg, x0, acts, th)
    out = np.zeros_like(emu)
    x0c, ac, tc = (np.ascontiguousarray(a, dtype=np.float64) for a in (x0, acts, th))
    rc = _lib.hostemu_lib().spi_hostemu_rollout_aba(ctypes.byref(r), x0c.ctypes.data, ac.ctypes.data,
                                                    tc.ctypes.data, x0.shape[0], acts.shape[1], out.ctypes.data)
    assert rc == 0
    assert np.abs(emu - out).max() < 1e-9


@pytest.mark.parametrize("kw", [dict(), dict(torque_speed=False), dict(tanh_a=(15.0, 18.0, 25.0), hip_action_scale=0.5),
                                dict(base_contact=False, motor_gain=(0.9, 1.1, 1.05))])
def test_hip_frame_legs_equal_articulated_body_algorithm(built, kw):
    """The legs condensed in the hip frame (csrc/leg_hip.cuh) and the oracle's articulated-body
    algorithm, both in FP64 with the same constants, agree to rounding: feet in and out of contact,
    base-box corners on the ground, each motor model."""
    from spi_gb300 import _lib, robot
    _, x0, acts, th = _inputs(16, B=24, H=12)
    x0[:8, 2] = 0.26
    x0[8:12, 2] = 0.08
    r = robot.to_struct(robot.SimConfig(**kw))
    x0c, ac, tc = (np.ascontiguousarray(a, dtype=np.float64) for a in (x0, acts, th))
    out = []
    for form in ("aba", "hip"):
        o = np.zeros((24, 12, 37))
        fn = getattr(_lib.hostemu_lib(), f"spi_hostemu_rollout_{form}")
        assert fn(ctypes.byref(r), x0c.ctypes.data, ac.ctypes.data, tc.ctypes.data, 24, 12, o.ctypes.data) == 0
        out.append(o)
    assert np.abs(out[0] - out[1]).max() < 1e-9


@pytest.mark.parametrize("kw", [dict(), dict(torque_speed=False, inertia_follows_mass=True),
                                dict(tanh_a=(15.0, 18.0, 25.0), motor_gain=(0.9, 1.1, 1.05))])
def test_substep_tangents_equal_central_differences(built, kw):
    """The substep tangents (csrc/tangent.cuh) in FP64 against central differences of the rollout (h = 1e-6:
    truncation and rounding each some 1e-9 of entries up to 1e2, hence 1e-4 with room for the curvature of
    contacts): feet in and out of contact, a base on the ground, saturated motors."""
    from spi_gb300 import _lib, robot
    _, x0, acts, th = _inputs(21, B=6, H=8)
    x0[3:5, 2] = 0.26
    x0[5, 2] = 0.06
    acts[4] *= 30
    r, lib = robot.to_struct(robot.SimConfig(**kw)), _lib.hostemu_lib()
    x0, acts, th = (np.ascontiguousarray(a, dtype=np.float64) for a in (x0, acts, th))
    for b in range(6):
        for k in range(13):
            state, d, ends = np.zeros(37), np.zeros(37), np.zeros((2, 8, 37))
            assert lib.spi_hostemu_tangent(ctypes.byref(r), x0[b].ctypes.data, acts[b].ctypes.data, th[b].ctypes.data, k, 8,
                                           state.ctypes.data, d.ctypes.data) == 0
            two = np.stack([th[b], th[b]])
            two[:, k] += (1e-6, -1e-6)
            x, a = np.stack([x0[b]] * 2), np.stack([acts[b]] * 2)
            assert lib.spi_hostemu_rollout(ctypes.byref(r), x.ctypes.data, a.ctypes.data, two.ctypes.data, 2, 8,
                                           ends.ctypes.data) == 0
            ref = (ends[0, -1] - ends[1, -1]) / 2e-6
            assert np.linalg.norm(d - ref) <= 1e-4 * max(np.linalg.norm(ref), 1e-2), (b, k)


def _f32p(*a):
    return [np.ascontiguousarray(x, dtype=np.float32) for x in a]


@pytest.mark.parametrize("vz", [-1.0, -0.5, 0.25])
def test_contact_tangent_at_a_speed_that_rounds_to_zero(built, vz):
    """The branch comes from the pass that produced the trajectory, the tangential velocity is formed again and
    may come out as exactly zero where that pass saw some. A foot that is off and slipping has no friction
    and none of its derivative; one that is on and slipping takes the sticking value, the model's at rest; one
    that is sticking keeps its damping, on or off. All exact in these numbers."""
    from spi_gb300 import _lib, robot
    cfg = robot.SimConfig()
    r, lib = robot.to_struct(cfg), _lib.hostemu_lib()
    v, n, dv, dn = _f32p([0, 0, vz], [0, 0, 1], [1, 2, 0], [0, 0, 0])

    def tan(z, on, stick):
        out = np.zeros(4, dtype=np.float32)
        assert lib.spi_hostemu_contact_tan(ctypes.byref(r), z, v.ctypes.data, n.ctypes.data, on, stick, 0.0,
                                           dv.ctypes.data, dn.ctypes.data, out.ctypes.data) == 0
        return out
    ct = np.float32(r.contact_ct)
    assert np.array_equal(tan(0.3, 0, 0), [0, 0, 0, 0])
    assert np.array_equal(tan(0.3, 0, 1), [-ct, -2 * ct, 0, 0])
    assert np.array_equal(tan(0.0, 1, 0), tan(0.0, 1, 1)) and np.isfinite(tan(0.0, 1, 1)).all()


def test_corner_tangent_takes_the_force_models_branch(built):
    """A base corner whose normal force (here some 1e-6 N) is far below its implicit mass's share of gravity (1e4 N), which
    it is added to: sliding at 1e-13 m/s it sticks (ct v < mu f), so a change of the velocity along x changes
    the force by -ct. The velocities leave a level base's other terms at zero, and ct is exact."""
    from spi_gb300 import _lib, robot
    r, lib = robot.to_struct(robot.SimConfig(contact_ct=2e6)), _lib.hostemu_lib()
    pen = np.float32(0.5) * np.float32(r.contact_ramp)
    corner = np.array(r.corners[0][:], dtype=np.float32)
    z = np.float32(-pen - corner[2])
    pen = float(np.float32(0) - np.float32(z + corner[2]))
    s = float(np.float32(pen) * np.float32(1.0 / np.float32(r.contact_ramp)))
    # a vertical velocity at which k pen and c s vz agree to within FP32 rounding, force just above zero
    vz = np.float32(r.contact_k * pen / (r.contact_c * s))
    for _ in range(64):
        f = np.float32(np.float32(r.contact_k) * np.float32(pen)) - np.float32(np.float32(np.float32(r.contact_c) * np.float32(s)) * vz)
        if f > 0:
            break
        vz = np.nextafter(vz, np.float32(0))
    assert 0 < f < 1e-4
    assert r.contact_ct * 1e-13 < r.contact_mu * f
    v, dv = _f32p([1e-13, 0, vz], [1, 0, 0])
    out = np.zeros(6, dtype=np.float32)
    assert lib.spi_hostemu_corner_tan(ctypes.byref(r), 0, 0, float(z), v.ctypes.data, dv.ctypes.data, out.ctypes.data) == 0
    assert out[3] == np.float32(r.contact_ct)


def test_kernel_vs_oracle_with_urdf_constants(built):
    """Float32 model constants move states by < 1e-5 (well inside the 1e-4 parity bar)."""
    cfg, x0, acts, th = _inputs(13)
    emu, _ = _emu(built, cfg, x0, acts, th)
    ref = dyn.rollout(x0, acts, th, gm.SimParams(), trace=True)
    err = np.abs(emu - ref) / np.maximum(np.abs(ref), 1.0)
    assert err.max() < 1e-5


def test_flop_count_constant(built):
    from spi_gb300 import _lib, robot
    cfg, x0, acts, th = _inputs(14, B=1, H=1)
    r = robot.to_struct(cfg)
    n1, n2 = ctypes.c_longlong(), ctypes.c_longlong()
    x0c = np.ascontiguousarray(x0[0], dtype=np.float64)
    tc = np.ascontiguousarray(th[0], dtype=np.float64)
    ac = np.ascontiguousarray(acts[0, 0], dtype=np.float64)
    lib = _lib.hostemu_lib()
    rc = lib.spi_hostemu_count_ops_aba(ctypes.byref(r), x0c.ctypes.data, tc.ctypes.data,
                                       ac.ctypes.data, ctypes.byref(n1), ctypes.byref(n2))
    assert rc == 0
    assert n1.value == FLOPS_PER_SUBSTEP
    rc = lib.spi_hostemu_count_ops(ctypes.byref(r), x0c.ctypes.data, tc.ctypes.data,
                                   ac.ctypes.data, ctypes.byref(n1), ctypes.byref(n2))
    assert rc == 0
    assert n1.value == EXECUTED_FLOPS_PER_SUBSTEP
    from spi_gb300 import flops
    assert flops.flops_per_rollout_step(cfg) == cfg.decimation * FLOPS_PER_SUBSTEP
    assert flops.executed_flops_per_rollout_step(cfg) == cfg.decimation * EXECUTED_FLOPS_PER_SUBSTEP
