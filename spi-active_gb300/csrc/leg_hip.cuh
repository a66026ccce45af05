// leg_hip.cuh -- one leg condensed onto the base, worked out in the hip frame.
//
// The same quantities as phase A of dynamics.cuh (the leg's articulated inertia and bias force at
// the base, and the work record of phase C), from about a third fewer operations. Everything
// is expressed in hip axes about the hip joint's origin o0:
//   * the thigh joint lies on the hip's y axis, so its axis passes through o0 and the thigh moves
//     about o0 itself; thigh and calf joints turn about the same axis, so the calf is placed by
//     the absolute angle q1 + q2. No velocity, acceleration or force is carried from link to link;
//   * inertias are second moments J = sum m r r^T (rotational inertia tr(J) 1 - J): a rotation
//     about y costs two multiply-adds on the double angle, a shift one chain per entry;
//   * the bias force is classical Newton-Euler. A body's acceleration field is a(r) = a_o + W r
//     with W = [dw/dt]x + w w^T - |w|^2 1; along the leg W changes by four entries only (the
//     column of the common hinge direction is shared), so one product with the whole leg's
//     composite plus two sparse corrections replaces three per-body passes.
// Derivation of the correction: with Q the joint rate relative to the hip, dw/dt gains
// (-w_z Q, 0, w_x Q) and w gains (0, Q, 0), so W_00 and W_22 lose d = (w_y + Q)^2 - w_y^2, and
// W_10, W_12 gain 2 Q w_x, 2 Q w_z.
#pragma once

#include "dynamics.cuh"

namespace spi {

// A leg's constants as leg_condense reads them, four to a 16-byte slot; 13 slots, so that the four legs' copies of a slot
// start in different shared-memory banks.
template <class S> struct alignas(16) HipLeg {
  S x0, y0, y1, z2;            // hip origin (x0, y0, 0), thigh origin (0, y1, 0), calf origin (0, 0, z2)
  S kd[3], m0;                 // joint damping; hip mass
  S iv[3], m12;                // 1 / velocity limit (0: no limit); thigh + calf mass
  S h0x, h0y, h0z, m2;         // hip first moment; calf mass
  S J0xx, J0yy, J0zz, J0xy;    // hip second moments about o0
  S J0xz, J0yz, h1x, h1z;      // thigh about o0, thigh axes: first moment,
  S h1y, P1, D1, X1;           //   (Jxx + Jzz) / 2, (Jxx - Jzz) / 2, Jxz,
  S J1xy, J1yz, yy12, h2x;     //   Jxy, Jyz; Jyy of thigh (about o0) + calf (about its joint)
  S h2y, h2z, P2, D2;          // calf about its joint, calf axes: as the thigh
  S X2, J2xy, J2yz, hf2;       //   hf2 = (foot z)^2 / 2
  S c0x, c0y, c0z, c1x;        // the leg's two base-box corners
  S c1y, c1z, pad[2];
  S pad2[4];
};
static_assert(sizeof(HipLeg<float>) == 13 * 16, "HipLeg: 13 slots");

// The model of the evaluation kernels, by value in their parameter block. The legs' constants stay out of DevModel: every
// other kernel copies that one to shared memory, CTA by CTA (832 bytes more took step_kernel, four substeps long,
// from 8.3 to 8.9 us).
struct EvalModel : DevModel {
  HipLeg<float> hip[4];
};
static_assert(sizeof(DevModel) == 2064, "DevModel: what every CTA copies");

// The constants of `leg` from the public robot description (S = float on the device).
template <class S> inline HipLeg<S> hip_leg_constants(const spi_robot& r, int leg) {
  HipLeg<S> c = {};
  double m[3], h[3][3], J[3][6];   // second moments xx yy zz xy xz yz about each body's origin
  for (int k = 0; k < 3; ++k) {
    const int b = 3 * leg + k;
    const float* I = r.body_I[b];
    m[k] = r.body_mass[b];
    for (int i = 0; i < 3; ++i) {
      h[k][i] = r.body_h[b][i];
      J[k][i] = 0.5 * ((double)I[0] + I[1] + I[2]) - (double)I[i];
      J[k][3 + i] = -(double)I[3 + i];
    }
    c.kd[k] = (S)((double)r.kd_scale * r.kd[b]);
    c.iv[k] = r.torque_speed ? (S)(1.0 / (double)r.velocity_limit[b]) : (S)0;
  }
  const double y1 = r.body_origin[3 * leg + 1][1], fz = r.foot[2];
  // the thigh moved out along the hip's y axis
  J[1][1] += 2.0 * h[1][1] * y1 + m[1] * y1 * y1;
  J[1][3] += h[1][0] * y1;
  J[1][5] += h[1][2] * y1;
  h[1][1] += m[1] * y1;
  c.x0 = (S)r.body_origin[3 * leg][0];
  c.y0 = (S)r.body_origin[3 * leg][1];
  c.y1 = (S)y1;
  c.z2 = (S)r.body_origin[3 * leg + 2][2];
  c.m0 = (S)m[0];
  c.m12 = (S)(m[1] + m[2]);
  c.m2 = (S)m[2];
  c.h0x = (S)h[0][0]; c.h0y = (S)h[0][1]; c.h0z = (S)h[0][2];
  c.J0xx = (S)J[0][0]; c.J0yy = (S)J[0][1]; c.J0zz = (S)J[0][2];
  c.J0xy = (S)J[0][3]; c.J0xz = (S)J[0][4]; c.J0yz = (S)J[0][5];
  c.h1x = (S)h[1][0]; c.h1y = (S)h[1][1]; c.h1z = (S)h[1][2];
  c.P1 = (S)(0.5 * (J[1][0] + J[1][2])); c.D1 = (S)(0.5 * (J[1][0] - J[1][2])); c.X1 = (S)J[1][4];
  c.J1xy = (S)J[1][3]; c.J1yz = (S)J[1][5];
  c.yy12 = (S)(J[1][1] + J[2][1]);
  c.h2x = (S)h[2][0]; c.h2y = (S)h[2][1]; c.h2z = (S)h[2][2];
  c.P2 = (S)(0.5 * (J[2][0] + J[2][2])); c.D2 = (S)(0.5 * (J[2][0] - J[2][2])); c.X2 = (S)J[2][4];
  c.J2xy = (S)J[2][3]; c.J2yz = (S)J[2][5];
  c.hf2 = (S)(0.5 * fz * fz);
  const float* k0 = r.corners[2 * leg];
  const float* k1 = r.corners[2 * leg + 1];
  c.c0x = (S)k0[0]; c.c0y = (S)k0[1]; c.c0z = (S)k0[2];
  c.c1x = (S)k1[0]; c.c1y = (S)k1[1]; c.c1z = (S)k1[2];
  return c;
}

// Rotation about x by (c, s) of a vector in the y-z plane: active (hip to base) and its transpose.
template <class T> SPI_INL V3<T> hip_to_base(T c, T s, T x, T y, T z) { return v3(x, c * y - s * z, s * y + c * z); }
template <class T> SPI_INL V3<T> base_to_hip(T c, T s, V3<T> u) { return v3(u.x, c * u.y + s * u.z, c * u.z - s * u.y); }

// Motor torque of a joint (motor_torque_at of dynamics.cuh on a leg's own constants).
template <int MS, class T>
SPI_INL T hip_motor(const DevModel& M, T kp, T lim, T fc, T kd, T iv, int k, T target, T q, T qd) {
  T tau = kp * (target - q) - kd * qd;
  if (MS == kMotorSpeedLimit || M.torque_speed) lim = lim * m_fmax(T(0), T(1) - m_fabs(qd) * iv);
  tau = m_clamp(tau, -lim, lim);
  if (MS == kMotorRuntime) {
    tau = tau * T(M.gain[k]);
    if (M.tanh_a[k] > 0.0f) tau = T(M.tanh_a[k]) * m_tanh(tau / T(M.tanh_a[k]));
    pin_device(tau);
  }
  return tau - fc * m_tanh_div(qd, M.fric_vel, M.fric_k2);
}

// The leg's contribution to the base: articulated inertia and bias force (out), and the work
// record of phase C (W.put_col, as phase_a_core). c: the leg's constants, P: its gains, tgt: the
// joint targets, corners: corners_may_touch(M, B).
template <int MS, class T, class S, class WK>
SPI_INL void leg_condense(const DevModel& M, const HipLeg<S>& c, const BaseState<T>& B, const LegState<T>& L,
                          const LegGains<T>& P, const T tgt[3], WK& W, LegOut<T>& out, bool corners) {
  const T qd0 = L.qd[0], qd1 = L.qd[1], qd2 = L.qd[2];
  T s0, c0, s1, c1, sk, ck;
  m_sincos(L.q[0], &s0, &c0);
  m_sincos(L.q[1], &s1, &c1);
  m_sincos(L.q[2], &sk, &ck);
  // the calf's absolute angle, composed: the error of the fast sine is then phase A's, joint by joint
  const T s2 = s1 * ck + c1 * sk, c2 = c1 * ck - s1 * sk;
  const T x0 = T(c.x0), y0 = T(c.y0), y1 = T(c.y1), z2 = T(c.z2), fz = T(M.foot[2]);

  // hip frame: base angular velocity w, velocity v and classical acceleration a of o0
  const V3<T> w = base_to_hip(c0, s0, B.nu.w);
  const V3<T> v = base_to_hip(c0, s0, v3(B.nu.v.x - B.nu.w.z * y0, B.nu.v.y + B.nu.w.z * x0,
                                         B.nu.v.z + B.nu.w.x * y0 - B.nu.w.y * x0));
  const V3<T> a = cross(w, v);
  const T wX = w.x + qd0, wy1 = w.y + qd1, wy2 = wy1 + qd2;

  // calf joint o2 = (x2, y1, zc), foot (px, y1, pz)
  const T x2 = z2 * s1, zc = z2 * c1, dx = fz * s2, dz = fz * c2;
  const T px = x2 + dx, pz = zc + dz;

  // foot contact, in hip axes; the implicit point mass takes part in the calf's Newton-Euler terms
  // below, where only its spatial acceleration belongs: the difference w x v_f is put back
  const V3<T> g0 = row(B.R, 2);
  const V3<T> g1 = base_to_hip(c0, s0, g0);
  const T zf = B.p.z + g0.x * x0 + g0.y * y0 + g1.x * px + g1.y * y1 + g1.z * pz;
  const V3<T> vf = v3(v.x - w.z * y1 + wy1 * zc + wy2 * dz, v.y + w.z * px - wX * pz,
                      v.z + wX * y1 - wy1 * x2 - wy2 * dx);
  T mimp;
  V3<T> Fc = contact_force_local(M, T(M.foot_r), zf, vf, g1, &mimp);
  Fc = cross_acc(mimp * v3(wX, wy2, w.z), vf, Fc);

  // calf (with the point mass) about its joint, in hip axes: first moment b, second moments E
  V3<T> b;
  S3<T> E;          // E.yy is a constant, folded into yy12
  T Eyy2;           // rotational inertia about the joint axis, E.xx + E.zz
  const T m2 = T(c.m2) + mimp;
  {
    const T hz = T(c.h2z) + mimp * fz, e = mimp * T(c.hf2);
    const T Pc = T(c.P2) + e, Dc = T(c.D2) - e;
    b = v3(c2 * T(c.h2x) + s2 * hz, T(c.h2y), c2 * hz - s2 * T(c.h2x));
    const T t2 = s2 + s2, sn = t2 * c2, cn = T(1) - t2 * s2;
    const T t = Dc * cn + T(c.X2) * sn;
    E.xx = Pc + t; E.zz = Pc - t; E.xz = T(c.X2) * cn - Dc * sn;
    E.xy = c2 * T(c.J2xy) + s2 * T(c.J2yz);
    E.yz = c2 * T(c.J2yz) - s2 * T(c.J2xy);
    Eyy2 = Pc + Pc;
  }
  // thigh + calf about o0: mass, first moment h, second moments J
  const T m1 = T(c.m12) + mimp;
  V3<T> h;
  S3<T> J;
  {
    const V3<T> hc = v3(b.x + m2 * x2, b.y + m2 * y1, b.z + m2 * zc);
    const T t2 = s1 + s1, sn = t2 * c1, cn = T(1) - t2 * s1;
    const T t = T(c.D1) * cn + T(c.X1) * sn;
    h = v3(hc.x + c1 * T(c.h1x) + s1 * T(c.h1z), hc.y + T(c.h1y), hc.z + c1 * T(c.h1z) - s1 * T(c.h1x));
    J.xx = E.xx + (T(c.P1) + t) + b.x * x2 + x2 * hc.x;
    J.zz = E.zz + (T(c.P1) - t) + b.z * zc + zc * hc.z;
    J.yy = T(c.yy12) + b.y * y1 + y1 * hc.y;
    J.xz = E.xz + T(c.X1) * cn - T(c.D1) * sn + b.x * zc + x2 * hc.z;
    J.xy = E.xy + c1 * T(c.J1xy) + s1 * T(c.J1yz) + b.x * y1 + x2 * hc.y;
    J.yz = E.yz + c1 * T(c.J1yz) - s1 * T(c.J1xy) + b.z * y1 + zc * hc.y;
  }
  // the whole leg about o0
  const T m = T(c.m0) + m1;
  const V3<T> H = v3(h.x + T(c.h0x), h.y + T(c.h0y), h.z + T(c.h0z));
  S3<T> G;
  G.xx = J.xx + T(c.J0xx); G.yy = J.yy + T(c.J0yy); G.zz = J.zz + T(c.J0zz);
  G.xy = J.xy + T(c.J0xy); G.xz = J.xz + T(c.J0xz); G.yz = J.yz + T(c.J0yz);

  // bias force (base and joint accelerations zero) on the leg about o0: F, N; joint torques n0, n1, n2
  V3<T> F, N;
  T n1, n2;
  {
    const T pX = wX + qd0;
    const T wxx = wX * wX, wyy = w.y * w.y, wzz = w.z * w.z, wyz = w.y * w.z;
    const T o01 = w.y * pX, o02 = w.z * pX, o10 = w.y * w.x, o20 = w.z * w.x;
    const T o00 = -wyy - wzz, o11 = -wxx - wzz, o22 = -wxx - wyy, dzx = wxx - wzz;
    const T d1 = qd1 * (wy1 + w.y), T1 = qd1 + qd1, d2 = qd2 * (wy2 + wy1), T2 = qd2 + qd2;
    // the calf's correction, a force f at its joint
    const V3<T> f = v3(-(d2 * b.x), T2 * (wX * b.x + w.z * b.z), -(d2 * b.z));
    F.x = f.x + m * a.x + o00 * H.x + o01 * H.y + o02 * H.z - d1 * h.x - Fc.x;
    F.y = f.y + m * a.y + o10 * H.x + o11 * H.y + wyz * H.z + T1 * (wX * h.x + w.z * h.z) - Fc.y;
    F.z = f.z + m * a.z + o20 * H.x + wyz * H.y + o22 * H.z - d1 * h.z - Fc.z;
    N.x = H.y * a.z - H.z * a.y + o20 * G.xy - o10 * G.xz + (wzz - wyy) * G.yz + wyz * (G.yy - G.zz)
          - d1 * J.yz - T1 * (wX * J.xz + w.z * J.zz) - d2 * E.yz - T2 * (wX * E.xz + w.z * E.zz)
          + y1 * f.z - zc * f.y - y1 * Fc.z + pz * Fc.y;
    N.z = H.x * a.y - H.y * a.x + (wyy - wxx) * G.xy + o10 * G.xx - o01 * G.yy + wyz * G.xz - o02 * G.yz
          + T1 * (wX * J.xx + w.z * J.xz) + d1 * J.xy + T2 * (wX * E.xx + w.z * E.xz) + d2 * E.xy
          + x2 * f.y - y1 * f.x - px * Fc.y + y1 * Fc.x;
    // thigh + calf about the y axis, then the hip's own share; the calf about its joint
    n1 = h.z * a.x - h.x * a.z + dzx * J.xz + o01 * J.yz - wyz * J.xy + o02 * J.zz - o20 * J.xx
         + zc * f.x - x2 * f.z - pz * Fc.x + px * Fc.z;
    N.y = n1 + T(c.h0z) * a.x - T(c.h0x) * a.z + dzx * T(c.J0xz) + o01 * T(c.J0yz) - wyz * T(c.J0xy)
          + o02 * T(c.J0zz) - o20 * T(c.J0xx);
    const T ax = a.x + (o00 - d1) * x2 + o01 * y1 + o02 * zc;    // acceleration of the calf joint
    const T az = a.z + o20 * x2 + wyz * y1 + (o22 - d1) * zc;
    n2 = b.z * ax - b.x * az + dzx * E.xz + o01 * E.yz - wyz * E.xy + o02 * E.zz - o20 * E.xx
         - dz * Fc.x + dx * Fc.z;
  }
  const T tau0 = hip_motor<MS>(M, P.kpk[0], P.lim[0], P.fc, T(c.kd[0]), T(c.iv[0]), 0, tgt[0], L.q[0], qd0);
  const T tau1 = hip_motor<MS>(M, P.kpk[1], P.lim[1], P.fc, T(c.kd[1]), T(c.iv[1]), 1, tgt[1], L.q[1], qd1);
  const T tau2 = hip_motor<MS>(M, P.kpk[2], P.lim[2], P.fc, T(c.kd[2]), T(c.iv[2]), 2, tgt[2], L.q[2], qd2);

  // joint force columns about o0 in hip axes, joint-space inertia M = L D L^T, and
  // K = F L^-T. F0 = (k0w; 0, -H.z, H.y), F1 = (-J.xy, J.xx + J.zz, -J.yz; h.z, 0, -h.x),
  // F2 = (.., Eyy2 + x2 b.x + zc b.z, ..; b.z, 0, -b.x)
  const T M00 = G.yy + G.zz, M01 = -J.xy, f1y = J.xx + J.zz;
  const T M02 = -E.xy - y1 * b.x, f2y = Eyy2 + x2 * b.x + zc * b.z, f2z = -E.yz - y1 * b.z;
  const T i0 = T(1) / (M00 + P.arm);
  const T l10 = M01 * i0, l20 = M02 * i0;
  const T i1 = T(1) / (f1y + P.arm - l10 * M01);
  const T e12 = f2y - l20 * M01;
  const T l21 = e12 * i1;
  const T i2 = T(1) / (Eyy2 + P.arm - l20 * M02 - l21 * e12);
  const T r1y = f1y + l10 * G.xy, r1z = l10 * G.xz - J.yz;               // F1.w - l10 F0.w, F0.w = (M00, -G.xy, -G.xz)
  const T r1x = M01 - l10 * M00;
  const T u1y = l10 * H.z, u1z = -h.x - l10 * H.y;                       // F1.v - l10 F0.v
  const V3<T> K2w = v3(M02 - l20 * M00 - l21 * r1x, f2y + l20 * G.xy - l21 * r1y, f2z + l20 * G.xz - l21 * r1z);
  const V3<T> K2v = v3(b.z - l21 * h.z, l20 * H.z - l21 * u1y, -b.x - l20 * H.y - l21 * u1z);
  // to base axes and the base origin: K0.v.x = 0
  SV<T> K0, K1, K2;
  {
    const V3<T> v0 = hip_to_base(c0, s0, T(0), -H.z, H.y), w0 = hip_to_base(c0, s0, M00, -G.xy, -G.xz);
    K0.v = v3(T(0), v0.y, v0.z);
    K0.w = v3(w0.x + y0 * v0.z, w0.y - x0 * v0.z, w0.z + x0 * v0.y);
    const V3<T> w1 = hip_to_base(c0, s0, r1x, r1y, r1z), w2 = hip_to_base(c0, s0, K2w.x, K2w.y, K2w.z);
    K1.v = hip_to_base(c0, s0, h.z, u1y, u1z);
    K1.w = add_rcross<kHipRM>(w1, v3(x0, y0, T(0)), K1.v);
    K2.v = hip_to_base(c0, s0, K2v.x, K2v.y, K2v.z);
    K2.w = add_rcross<kHipRM>(w2, v3(x0, y0, T(0)), K2.v);
  }
  SV<T> Kp0;
  Kp0.w = i0 * K0.w;
  Kp0.v = v3(T(0), i0 * K0.v.y, i0 * K0.v.z);
  const SV<T> Kp1 = i1 * K1, Kp2 = i2 * K2;
  const T t0 = tau0 - N.x;
  const T t1 = (tau1 - n1) - l10 * t0;
  const T t2 = (tau2 - n2) - l20 * t0 - l21 * t1;
  const T e0 = t0 * i0, e1 = t1 * i1, e2 = t2 * i2;
  W.put_col(0, Kp0, e0, l10);
  W.put_col(1, Kp1, e1, l20);
  W.put_col(2, Kp2, e2, l21);

  // the leg at the base: rigid inertia less K D^-1 K^T, bias + K y
  {
    const T t2a = s0 + s0, sn = t2a * c0, cn = T(1) - t2a * s0;
    const T hs = T(0.5) * (G.yy + G.zz), hd = T(0.5) * (G.yy - G.zz);
    const T t = hd * cn - G.yz * sn;
    const V3<T> Hb = hip_to_base(c0, s0, H.x, H.y, H.z);
    const V3<T> Hr = v3(Hb.x + m * x0, Hb.y + m * y0, Hb.z);
    const T xx = G.xx + Hb.x * x0 + x0 * Hr.x, yy = (hs + t) + Hb.y * y0 + y0 * Hr.y, zz = hs - t;
    out.I.A.xx = yy + zz; out.I.A.yy = xx + zz; out.I.A.zz = xx + yy;
    out.I.A.xy = s0 * G.xz - c0 * G.xy - Hb.x * y0 - x0 * Hr.y;
    out.I.A.xz = -(s0 * G.xy) - c0 * G.xz - x0 * Hr.z;
    out.I.A.yz = -(hd * sn) - G.yz * cn - y0 * Hr.z;
    out.I.B.m[0][0] = T(0); out.I.B.m[0][1] = -Hr.z; out.I.B.m[0][2] = Hr.y;
    out.I.B.m[1][0] = Hr.z; out.I.B.m[1][1] = T(0); out.I.B.m[1][2] = -Hr.x;
    out.I.B.m[2][0] = -Hr.y; out.I.B.m[2][1] = Hr.x; out.I.B.m[2][2] = T(0);
    out.I.C.xx = m; out.I.C.yy = m; out.I.C.zz = m; out.I.C.xy = T(0); out.I.C.xz = T(0); out.I.C.yz = T(0);
  }
  art_sub_outer(out.I, Kp2, K2);
  art_sub_outer(out.I, Kp1, K1);
  art_sub_outer_vx0(out.I, Kp0, K0);
  const V3<T> pv = hip_to_base(c0, s0, F.x, F.y, F.z);
  const V3<T> pw = add_rcross<kHipRM>(hip_to_base(c0, s0, N.x, N.y, N.z), v3(x0, y0, T(0)), pv);
  out.p.w = v3(pw.x + e2 * K2.w.x + e1 * K1.w.x + e0 * K0.w.x, pw.y + e2 * K2.w.y + e1 * K1.w.y + e0 * K0.w.y,
               pw.z + e2 * K2.w.z + e1 * K1.w.z + e0 * K0.w.z);
  out.p.v = v3(pv.x + e2 * K2.v.x + e1 * K1.v.x, pv.y + e2 * K2.v.y + e1 * K1.v.y + e0 * K0.v.y,
               pv.z + e2 * K2.v.z + e1 * K1.v.z + e0 * K0.v.z);
  if (corners) {   // two of the eight base-box corners (as phase_a_core)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const V3<T> rc = j == 0 ? v3(T(c.c0x), T(c.c0y), T(c.c0z)) : v3(T(c.c1x), T(c.c1y), T(c.c1z));
      const V3<T> vc = cross_acc(B.nu.w, rc, B.nu.v);
      T mc;
      V3<T> Fw = contact_force(M, T(0), B.p.z + B.R.m[2][0] * rc.x + B.R.m[2][1] * rc.y + B.R.m[2][2] * rc.z,
                               mul(B.R, vc), &mc);
      Fw.z = Fw.z + mc * T(M.g);
      const V3<T> Fb = mulT(B.R, Fw);
      out.p.w = cross_acc(Fb, rc, out.p.w);
      out.p.v = out.p.v - Fb;
      add_point_mass(out.I, mc, rc);
    }
  }
}

}  // namespace spi
