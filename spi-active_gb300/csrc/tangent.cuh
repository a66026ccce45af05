// tangent.cuh -- one physics substep's forward tangent from the equations of motion.
//
// A substep's accelerations a = (a0, qdd) solve r(x, theta, a) = 0 (adjoint.cuh), so a direction
// (dx, dtheta) moves them by da = -M'^-1 dr with dr = (dr/dx) dx + (dr/dtheta) dtheta at fixed a. Given the
// substep's factorisation, a direction costs the tangent of the recursive Newton-Euler residual and
// two triangular solves: 8,564 operations a substep with the residual itself (5,152 where directions
// share that) against 15,969 for carrying the direction through the condensation and the Cholesky
// factorisation. Each function below is the derivative of the function of the same name in
// adjoint.cuh / dynamics.cuh; for a motion o = X m across a joint, do = X dm + (o x S) dq.
//
// The contact's branches (normal force on or off, stick or slip) are given, not decided here: the pass
// that produced the trajectory hands them over with the foot height, so that the tangent is
// that of the branch it took.
#pragma once

#include "adjoint.cuh"

namespace spi {
namespace tng {

template <class T> struct BaseTan {   // tangent of the base state; R's follows from the quaternion's
  V3<T> p;
  T qx, qy, qz, qw;
  SV<T> nu;
  M3<T> R;
};
template <class T> struct LegTan { T q[3], qd[3]; };
// Tangents of the parameters: base rigid inertia and the leg's motor terms.
template <class T> struct ParamTan { T m; V3<T> h; S3<T> Io; T kps, fc, arm, ts; };

struct ContactBranch { bool on, stick; };

// d quat_to_R along (x, y, z, w)' = d.
template <class T> SPI_INL M3<T> quat_to_R_tan(T x, T y, T z, T w, T dx, T dy, T dz, T dw) {
  M3<T> R;
  R.m[0][0] = T(-4) * (y * dy + z * dz);
  R.m[1][1] = T(-4) * (x * dx + z * dz);
  R.m[2][2] = T(-4) * (x * dx + y * dy);
  R.m[0][1] = T(2) * (x * dy + y * dx - z * dw - w * dz);
  R.m[1][0] = T(2) * (x * dy + y * dx + z * dw + w * dz);
  R.m[0][2] = T(2) * (x * dz + z * dx + y * dw + w * dy);
  R.m[2][0] = T(2) * (x * dz + z * dx - y * dw - w * dy);
  R.m[1][2] = T(2) * (y * dz + z * dy - x * dw - w * dx);
  R.m[2][1] = T(2) * (y * dz + z * dy + x * dw + w * dx);
  return R;
}

// The base rigid inertia's tangent (base_params) along theta slot k < 5; zero for the others.
template <class T> SPI_INL void base_params_tan(const DevModel& M, const T* th, int k, T& dm, V3<T>& dh, S3<T>& dI) {
  const T m = th[0];
  const V3<T> c = v3(T(M.base_com[0]) + th[1], T(M.base_com[1]) + th[2], T(M.base_com[2]) + th[3]);
  const T f = M.inertia_follows_mass ? m / T(M.base_m0) : T(1);
  dm = k == 0 ? T(1) : T(0);
  const V3<T> dc = v3(k == 1 ? T(1) : T(0), k == 2 ? T(1) : T(0), k == 3 ? T(1) : T(0));
  const T df = k == 0 && M.inertia_follows_mass ? T(1) / T(M.base_m0) : T(0);
  const T ds = k == 4 ? T(1) : T(0);
  dh = dm * c + m * dc;
  const T g = df * th[4] + f * ds;
  const T cc = dot(c, c), cdc = T(2) * dot(c, dc);
  dI.xx = g * T(M.base_Ic[0]) + dm * (cc - c.x * c.x) + m * (cdc - T(2) * c.x * dc.x);
  dI.yy = g * T(M.base_Ic[1]) + dm * (cc - c.y * c.y) + m * (cdc - T(2) * c.y * dc.y);
  dI.zz = g * T(M.base_Ic[2]) + dm * (cc - c.z * c.z) + m * (cdc - T(2) * c.z * dc.z);
  dI.xy = df * T(M.base_Ic[3]) - dm * c.x * c.y - m * (dc.x * c.y + c.x * dc.y);
  dI.xz = df * T(M.base_Ic[4]) - dm * c.x * c.z - m * (dc.x * c.z + c.x * dc.z);
  dI.yz = df * T(M.base_Ic[5]) - dm * c.y * c.z - m * (dc.y * c.z + c.y * dc.z);
}

// contact_force_local: dF and d mimp from dz, dv, dn on the given branch.
template <class T>
SPI_INL V3<T> contact_tan(const DevModel& M, T radius, T z, V3<T> v, V3<T> n, ContactBranch br, T dz, V3<T> dv, V3<T> dn,
                          T& dmimp) {
  const T vz = dot(n, v);
  const V3<T> vt = v3(v.x - vz * n.x, v.y - vz * n.y, v.z - vz * n.z);
  const T pen = radius - z, sarg = pen * T(M.ramp_inv);
  const T s = m_clamp(sarg, T(0), T(1));
  const T fn = br.on ? T(M.k) * pen - T(M.c) * s * vz : T(0);
  const T dmds = m_mul2_c(T(1), M.dt, M.imp_c, M.dt_imp_c);
  const T fz = fn + s * dmds * T(M.g);
  const T ds = sarg >= T(0) && sarg <= T(1) ? -(dz * T(M.ramp_inv)) : T(0);
  const T dvz = dot(dn, v) + dot(n, dv);
  const V3<T> dvt = v3(dv.x - dvz * n.x - vz * dn.x, dv.y - dvz * n.y - vz * dn.y, dv.z - dvz * n.z - vz * dn.z);
  const T dfn = br.on ? -(T(M.k) * dz) - T(M.c) * (ds * vz + s * dvz) : T(0);
  dmimp = dmds * ds;
  const T dfz = dfn + dmimp * T(M.g);
  // The branch is the forward pass's, vt is formed here, with other roundings: a slip's speed may come out as zero.
  // Off, a slip has no friction whatever its speed; on, the value at rest is the sticking one. (Selected, not branched
  // on: 4096 windows x 13 directions 1.53 ms, 1.57 with a branch.)
  const T vv = dot(vt, vt);
  const bool slides = br.on && !br.stick && vv > T(0);
  const T inv = T(1) / m_sqrt(vv);
  const T ss = T(M.mu) * fn * inv, dss = (T(M.mu) * dfn - ss * dot(vt, dvt) * inv) * inv;
  const T scale = slides ? ss : (br.stick || br.on ? T(M.ct) : T(0)), dscale = slides ? dss : T(0);
  return v3(dfz * n.x + fz * dn.x - dscale * vt.x - scale * dvt.x, dfz * n.y + fz * dn.y - dscale * vt.y - scale * dvt.y,
            dfz * n.z + fz * dn.z - dscale * vt.z - scale * dvt.z);
}

// motor_torque_at.
template <class T>
SPI_INL T motor_tan(const DevModel& M, const LegParams<T>& P, int k, int leg, T target, T q, T qd, T dq, T dqd, T dkps,
                    T dfc, T dts) {
  const F4* lc = M.legc[leg];
  const T Kp = T(M.kp[k][leg]), kp = P.kp_of(M, k, leg), e = target - q;
  const T kdk = m_mul2_c(T(1), M.kd_scale, M.kd[k][leg], lc[k].w);
  const T tau0 = kp * e - kdk * qd, lim0 = P.lim_of(M, k, leg);
  T lim = lim0, dlim = dts * T(M.tlim[k][leg]);
  if (M.torque_speed) {
    const T u = T(1) - m_div_c(m_fabs(qd), M.vlim[k][leg], lc[5 + 3 * k].z);
    const T du = m_div_c(qd >= T(0) ? -dqd : dqd, M.vlim[k][leg], lc[5 + 3 * k].z);
    const T sp = m_fmax(T(0), u);
    dlim = dlim * sp + (u > T(0) ? lim0 * du : T(0));
    lim = lim0 * sp;
  }
  T d = dkps * Kp * e - kp * dq - kdk * dqd, tau = tau0;
  if (tau0 > lim) { d = dlim; tau = lim; }
  else if (tau0 < -lim) { d = -dlim; tau = -lim; }
  d = d * T(M.gain[k]);
  if (M.tanh_a[k] > 0.0f) {
    const T t = m_tanh(tau * T(M.gain[k]) / T(M.tanh_a[k]));
    d = d * (T(1) - t * t);
  }
  const T tf = m_tanh_div(qd, M.fric_vel, M.fric_k2);
  return d - dfc * tf - P.fc * (T(1) - tf * tf) / T(M.fric_vel) * dqd;
}

// S x* f for the joint axis AX, times dq, added to df.
template <int AX, class T> SPI_INL SV<T> turn_force(const SV<T>& df, const SV<T>& f, T dq) {
  SV<T> o = df;
  if (AX == 0) { o.w.y -= f.w.z * dq; o.w.z += f.w.y * dq; o.v.y -= f.v.z * dq; o.v.z += f.v.y * dq; }
  else { o.w.x += f.w.z * dq; o.w.z -= f.w.x * dq; o.v.x += f.v.z * dq; o.v.z -= f.v.x * dq; }
  return o;
}
template <class T> SPI_INL SV<T> sv_sub(const SV<T>& a, const SV<T>& b) { return adj::sub_sv(a, b); }

// The residual's tangent of one leg (leg_residual): dr[3] and the force on the base dfb. t: the leg's tape at
// the substep (leg_pose, leg_residual); g0 = the tangent of the world vertical in base coordinates.
template <class T>
SPI_INL void leg_residual_tan(const DevModel& M, int leg, const BaseState<T>& B, const LegState<T>& L, const LegParams<T>& P,
                              const T tgt[3], const T qdd[3], const adj::LegTape<T>& t, T zf, ContactBranch br,
                              const BaseTan<T>& dB, const LegTan<T>& dL, const ParamTan<T>& dP, T dr[3], SV<T>& dfb) {
  const F4* lc = M.legc[leg];
  const V3<T> r0 = lc_org<T>(lc, 0), r1 = lc_org<T>(lc, 1), r2 = lc_org<T>(lc, 2);
  const T fz = T(M.foot[2]);
  const T *c = t.c, *s = t.s;
  const T dq0 = dL.q[0], dq1 = dL.q[1], dq2 = dL.q[2];
  // velocities and velocity products
  SV<T> dv0 = motion_to_child<0, kHipRM>(dB.nu, c[0], s[0], r0) + vel_product<0>(t.v0, dq0);
  dv0.w.x = dv0.w.x + dL.qd[0];
  SV<T> dv1 = motion_to_child<1, 2>(dv0, c[1], s[1], r1) + vel_product<1>(t.v1, dq1);
  dv1.w.y = dv1.w.y + dL.qd[1];
  SV<T> dv2 = motion_to_child<1, 4>(dv1, c[2], s[2], r2) + vel_product<1>(t.v2, dq2);
  dv2.w.y = dv2.w.y + dL.qd[2];
  // accelerations: al_k less its own velocity product is the parent's, carried over
  const SV<T> da0 = vel_product<0>(dv0, L.qd[0]) + vel_product<0>(t.v0, dL.qd[0]) +
                    vel_product<0>(sv_sub(t.al0, vel_product<0>(t.v0, L.qd[0])), dq0);
  const SV<T> da1 = motion_to_child<1, 2>(da0, c[1], s[1], r1) + vel_product<1>(dv1, L.qd[1]) + vel_product<1>(t.v1, dL.qd[1]) +
                    vel_product<1>(sv_sub(t.al1, vel_product<1>(t.v1, L.qd[1])), dq1);
  const SV<T> da2 = motion_to_child<1, 4>(da1, c[2], s[2], r2) + vel_product<1>(dv2, L.qd[2]) + vel_product<1>(t.v2, dL.qd[2]) +
                    vel_product<1>(sv_sub(t.al2, vel_product<1>(t.v2, L.qd[2])), dq2);
  // contact
  const V3<T> dg0 = row(dB.R, 2);
  V3<T> dg1 = rotT<0>(c[0], s[0], dg0);
  dg1.y = dg1.y + t.g1.z * dq0; dg1.z = dg1.z - t.g1.y * dq0;
  V3<T> dg2 = rotT<1>(c[1], s[1], dg1);
  dg2.x = dg2.x - t.g2.z * dq1; dg2.z = dg2.z + t.g2.x * dq1;
  V3<T> dg3 = rotT<1>(c[2], s[2], dg2);
  dg3.x = dg3.x - t.g3.z * dq2; dg3.z = dg3.z + t.g3.x * dq2;
  const T dzf = dB.p.z + dg0.x * r0.x + dg0.y * r0.y + dg1.y * r1.y + dg2.z * r2.z + dg3.z * fz;
  const V3<T> dvf = v3(dv2.v.x + dv2.w.y * fz, dv2.v.y - dv2.w.x * fz, dv2.v.z);
  T dmimp;
  const V3<T> dF = contact_tan(M, T(M.foot_r), zf, t.vf, t.g3, br, dzf, dvf, dg3, dmimp);
  // forces
  const RI<T> Ihp = lc_ri<T>(lc, 0), Ith = lc_ri<T>(lc, 1), Ical = lc_ri<T>(lc, 2);
  RI<T> Rc2 = Ical;
  {
    const T hz = t.mimp * fz;
    Rc2.m = Rc2.m + t.mimp;
    Rc2.h.z = Rc2.h.z + hz;
    Rc2.I.xx = Rc2.I.xx + hz * fz;
    Rc2.I.yy = Rc2.I.yy + hz * fz;
  }
  SV<T> df2 = ri_mul_acc(Rc2, da2, crf_acc(dv2, t.h2, crf(t.v2, ri_mul(Ical, dv2))));
  {   // d mimp times the point mass's share, and the contact force
    const V3<T> u = v3(t.al2.v.x + t.al2.w.y * fz, t.al2.v.y - t.al2.w.x * fz, t.al2.v.z);
    df2.v = v3(df2.v.x + dmimp * u.x - dF.x, df2.v.y + dmimp * u.y - dF.y, df2.v.z + dmimp * u.z - dF.z);
    df2.w.x = df2.w.x - fz * (dmimp * u.y - dF.y);
    df2.w.y = df2.w.y + fz * (dmimp * u.x - dF.x);
  }
  const SV<T> df1 = force_to_parent_acc<1, 4>(turn_force<1>(df2, t.f2, dq2), c[2], s[2], r2,
                                              ri_mul_acc(Ith, da1, crf_acc(dv1, t.h1, crf(t.v1, ri_mul(Ith, dv1)))));
  const SV<T> df0 = force_to_parent_acc<1, 2>(turn_force<1>(df1, t.f1, dq1), c[1], s[1], r1,
                                              ri_mul_acc(Ihp, da0, crf_acc(dv0, t.h0, crf(t.v0, ri_mul(Ihp, dv0)))));
  dfb = force_to_parent<0, kHipRM>(turn_force<0>(df0, t.f0, dq0), c[0], s[0], r0);
  const T fk[3] = {df0.w.x, df1.w.y, df2.w.y};
#pragma unroll
  for (int k = 0; k < 3; ++k)
    dr[k] = fk[k] + dP.arm * qdd[k] -
            motor_tan(M, P, k, leg, tgt[k], L.q[k], L.qd[k], dL.q[k], dL.qd[k], dP.kps, dP.fc, dP.ts);
}

// The base body's own residual terms.
template <class T>
SPI_INL SV<T> base_residual_tan(const BaseParams<T>& bp, const BaseState<T>& B, const SV<T>& a0, const BaseTan<T>& dB,
                                const ParamTan<T>& dP) {
  const SV<T> h = rigid_mul(bp.m, bp.h, bp.Io, B.nu);
  const SV<T> dh = rigid_mul_acc(dP.m, dP.h, dP.Io, B.nu, rigid_mul(bp.m, bp.h, bp.Io, dB.nu));
  return rigid_mul_acc(dP.m, dP.h, dP.Io, a0, crf_acc(dB.nu, h, crf(B.nu, dh)));
}

// One base-box corner's residual term P(mc, rc) a0 - (rc x Fb; Fb).
template <class T>
SPI_INL SV<T> corner_residual_tan(const DevModel& M, const BaseState<T>& B, V3<T> rc, const SV<T>& a0, const BaseTan<T>& dB) {
  const V3<T> ez = v3(T(0), T(0), T(1)), z0 = v3(T(0), T(0), T(0));
  const V3<T> vc = cross_acc(B.nu.w, rc, B.nu.v), dvc = cross_acc(dB.nu.w, rc, dB.nu.v);
  const V3<T> vw = mul(B.R, vc), dvw = mul(dB.R, vc) + mul(B.R, dvc);
  const T zc = B.p.z + dot(row(B.R, 2), rc), dz = dB.p.z + dot(row(dB.R, 2), rc);
  T mc, dmc, branch[2];
  const V3<T> F = contact_force_local(M, T(0), zc, vw, ez, &mc, branch);
  const ContactBranch br = {branch[0] > T(0), branch[1] == T(M.ct)};
  const V3<T> dF = contact_tan(M, T(0), zc, vw, ez, br, dz, dvw, z0, dmc);
  const V3<T> dFb = mulT(dB.R, F) + mulT(B.R, dF);
  const V3<T> u = dmc * cross_acc(a0.w, rc, a0.v) - dFb;     // rate of the point's force
  SV<T> o;
  o.v = u;
  o.w = cross(rc, u);
  return o;
}

// The integrator's tangent (base_solve's tail): B0 before, B1 after the substep, da0 the base acceleration's
// tangent; dB is advanced in place.
template <class T>
SPI_INL void base_integrate_tan(const DevModel& M, const BaseState<T>& B0, const BaseState<T>& B1, const SV<T>& da0,
                                BaseTan<T>& dB) {
  const T dt = T(M.dt), g = T(M.g), hx = T(0.5) * dt;
  dB.nu.w = dB.nu.w + dt * da0.w;
  dB.nu.v = dB.nu.v + dt * (da0.v - g * row(dB.R, 2));
  const V3<T> w = B1.nu.w, dw = dB.nu.w;
  const T nx = B0.qx + hx * (B0.qw * w.x + (B0.qy * w.z - B0.qz * w.y));
  const T ny = B0.qy + hx * (B0.qw * w.y + (B0.qz * w.x - B0.qx * w.z));
  const T nz = B0.qz + hx * (B0.qw * w.z + (B0.qx * w.y - B0.qy * w.x));
  const T nw = B0.qw - hx * (B0.qx * w.x + B0.qy * w.y + B0.qz * w.z);
  const T inv = T(1) / m_sqrt(nx * nx + ny * ny + nz * nz + nw * nw);
  const T dx = dB.qx + hx * (dB.qw * w.x + dB.qy * w.z - dB.qz * w.y + B0.qw * dw.x + B0.qy * dw.z - B0.qz * dw.y);
  const T dy = dB.qy + hx * (dB.qw * w.y + dB.qz * w.x - dB.qx * w.z + B0.qw * dw.y + B0.qz * dw.x - B0.qx * dw.z);
  const T dz = dB.qz + hx * (dB.qw * w.z + dB.qx * w.y - dB.qy * w.x + B0.qw * dw.z + B0.qx * dw.y - B0.qy * dw.x);
  const T dw4 = dB.qw - hx * (dB.qx * w.x + dB.qy * w.y + dB.qz * w.z + B0.qx * dw.x + B0.qy * dw.y + B0.qz * dw.z);
  const T pr = B1.qx * dx + B1.qy * dy + B1.qz * dz + B1.qw * dw4;
  dB.qx = (dx - B1.qx * pr) * inv;
  dB.qy = (dy - B1.qy * pr) * inv;
  dB.qz = (dz - B1.qz * pr) * inv;
  dB.qw = (dw4 - B1.qw * pr) * inv;
  dB.R = quat_to_R_tan(B1.qx, B1.qy, B1.qz, B1.qw, dB.qx, dB.qy, dB.qz, dB.qw);
  dB.p = dB.p + dt * (mul(dB.R, B1.nu.v) + mul(B1.R, dB.nu.v));
}

// The window's start (base_from_world) does not depend on theta; the final state's world-frame tangent.
template <class T> SPI_INL void base_to_world_tan(const BaseState<T>& B, const BaseTan<T>& dB, T* s13) {
  s13[0] = dB.p.x; s13[1] = dB.p.y; s13[2] = dB.p.z;
  s13[3] = dB.qx; s13[4] = dB.qy; s13[5] = dB.qz; s13[6] = dB.qw;
  const V3<T> v = mul(dB.R, B.nu.v) + mul(B.R, dB.nu.v), w = mul(dB.R, B.nu.w) + mul(B.R, dB.nu.w);
  s13[7] = v.x; s13[8] = v.y; s13[9] = v.z;
  s13[10] = w.x; s13[11] = w.y; s13[12] = w.z;
}
template <class T> SPI_INL BaseTan<T> zero_base_tan() {
  BaseTan<T> d;
  d.p = adj::z3<T>();
  d.qx = d.qy = d.qz = d.qw = T(0);
  d.nu = adj::zsv<T>();
  d.R = adj::zm3<T>();
  return d;
}

}  // namespace tng
}  // namespace spi
