// rollout_hip.cuh -- rollouts with the legs condensed in the hip frame (leg_hip.cuh): spi_run on a
// caller's theta batch.
//
// Two forms of one rollout, with the same bits:
//   lane  one lane carries a rollout through its four legs in turn (substep_hip_lane), the form that does
//         least work in total;
//   team  four lanes carry it, one leg each (TeamRollout), the form with the shortest chain: per
//         substep one leg, a sum through shared memory and the base solve, for launches that leave
//         schedulers idle.
// Both call the same functions on pinned inputs (pin: no multiply-add is fused across the
// value's definition) and add the base body's terms and the legs FL, FR, RL, RR in that order, so
// the choice does not show in the results.
#pragma once

#include <cuda_runtime.h>

#include "leg_hip.cuh"
#include "rollout_lane.cuh"

namespace spi {

// pin (dynamics.cuh) of the composite values handed from one function to the next.
__device__ __forceinline__ void pin3(V3<float>& v) { pin(v.x); pin(v.y); pin(v.z); }
__device__ __forceinline__ void pin_s3(S3<float>& s) {
  pin(s.xx); pin(s.yy); pin(s.zz); pin(s.xy); pin(s.xz); pin(s.yz);
}
__device__ __forceinline__ void pin(LegOut<float>& o) {
  pin_s3(o.I.A);
  pin_s3(o.I.C);
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) pin(o.I.B.m[i][j]);
  pin3(o.p.w);
  pin3(o.p.v);
}
__device__ __forceinline__ void pin(BaseState<float>& B) {
  pin3(B.p);
  pin(B.qx); pin(B.qy); pin(B.qz); pin(B.qw);
  pin3(B.nu.w);
  pin3(B.nu.v);
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) pin(B.R.m[i][j]);
}
__device__ __forceinline__ void pin(LegGains<float>& g) {
#pragma unroll
  for (int k = 0; k < 3; ++k) { pin(g.kpk[k]); pin(g.lim[k]); }
  pin(g.fc);
  pin(g.arm);
}
__device__ __forceinline__ void pin(LegWork<float>& W) {
#pragma unroll
  for (int k = 0; k < 3; ++k) { pin3(W.Kp[k].w); pin3(W.Kp[k].v); pin(W.y[k]); }
  pin(W.l10); pin(W.l20); pin(W.l21);
}
// Positions carry their rounding error (x + e is the sum): the integrator adds some 1e-4 m or rad a
// substep to values near 0.3 and 1.5, and the feet's 20 kN/m springs turn what rounds away into force.
// It halves the FP32 error of a window's cost (measured on the host: 2.4e-6 to 1.3e-6) for about 30
// of the substep's 2,900 instructions. The base position and the thigh and calf angles, which
// place the feet, are summed this way.
__device__ __forceinline__ void carry_add(float& x, float& e, float d) {
  const float y = d + e;
  const float t = x + y;
  e = y - (t - x);
  x = t;
}
__device__ __forceinline__ void carry_add(V3<float>& x, V3<float>& e, const V3<float>& d) {
  carry_add(x.x, e.x, d.x);
  carry_add(x.y, e.y, d.y);
  carry_add(x.z, e.z, d.z);
}
// Joint integration of a leg (phase_c) with the carried errors of q[1], q[2] in e.
template <class WK>
__device__ __forceinline__ void joint_step(const DevModel& M, const SV<float>& a0, const WK& W, LegState<float>& L,
                                           float e[2]) {
  float qdd[3];
  joint_accel(a0, W, qdd);
#pragma unroll
  for (int k = 0; k < 3; ++k) L.qd[k] = L.qd[k] + M.dt * qdd[k];
  L.q[0] = L.q[0] + M.dt * L.qd[0];
  carry_add(L.q[1], e[0], M.dt * L.qd[1]);
  carry_add(L.q[2], e[1], M.dt * L.qd[2]);
}

__device__ __forceinline__ void add_out(LegOut<float>& a, const LegOut<float>& b) {
  add_to(a.I, b.I);
  a.p.w = a.p.w + b.p.w;
  a.p.v = a.p.v + b.p.v;
}
// A leg's constants from the kernel's parameter block, sixteen bytes a load.
__device__ __forceinline__ HipLeg<float> load_hip(const HipLeg<float>* p) {
  HipLeg<float> c;
  const float4* s = reinterpret_cast<const float4*>(p);
  float4* d = reinterpret_cast<float4*>(&c);
#pragma unroll
  for (int i = 0; i < 12; ++i) d[i] = s[i];
  return c;
}

// One thread's shared-memory slots in the lane form, 16-byte fields [field][128 threads], each warp access
// one conflict-free 128-bit load or store: the legs' parked work records (kParkVec each), then per leg
// (q0, q1, q2, qd0), the joint targets (t0, t1, t2, 0) and (qd1, qd2, the errors of q1 and q2). 144 floats a
// thread, 72 KB a CTA: three CTAs (12 warps) per SM.
constexpr int kHipStateA = 4 * kParkVec;
constexpr int kHipTargets = kHipStateA + 4;
constexpr int kHipStateB = kHipTargets + 4;
constexpr int kHipSlotBytes = (kHipStateB + 4) * 128 * (int)sizeof(float4);
struct HipSlots {
  float4* sm;
  __device__ __forceinline__ float4& field(int f) const { return sm[f * 128]; }
  __device__ __forceinline__ float4* park(int leg) const { return sm + leg * kParkVec * 128; }
  __device__ __forceinline__ LegState<float> leg_state(int leg, float e[2]) const {
    const float4 u = field(kHipStateA + leg), v = field(kHipStateB + leg);
    LegState<float> L;
    L.q[0] = u.x; L.q[1] = u.y; L.q[2] = u.z;
    L.qd[0] = u.w; L.qd[1] = v.x; L.qd[2] = v.y;
    e[0] = v.z; e[1] = v.w;
    return L;
  }
  __device__ __forceinline__ void put_leg_state(int leg, const LegState<float>& L, const float e[2]) const {
    field(kHipStateA + leg) = make_float4(L.q[0], L.q[1], L.q[2], L.qd[0]);
    field(kHipStateB + leg) = make_float4(L.qd[1], L.qd[2], e[0], e[1]);
  }
  // the joint targets of the twelve actions of one control step (legs in order)
  __device__ __forceinline__ void put_targets(const DevModel& M, const float4 a0, const float4 a1, const float4 a2) const {
    const float a[12] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w, a2.x, a2.y, a2.z, a2.w};
    float t[12];
#pragma unroll
    for (int j = 0; j < 12; ++j) t[j] = joint_target(M, j % 3, j / 3, a[j]);
#pragma unroll
    for (int leg = 0; leg < 4; ++leg)
      field(kHipTargets + leg) = make_float4(t[3 * leg], t[3 * leg + 1], t[3 * leg + 2], 0.f);
  }
};

// One physics substep of one rollout on one lane. s: this thread's slots; bp: the warp's base
// parameters; gains: the warp's four legs' LegGains (two fields each); pe: the base position's error.
template <int MS>
__device__ __forceinline__ void substep_hip_lane(const EvalModel& M, BaseState<float>& B, V3<float>& pe, const HipSlots& s,
                                                 const BaseParams<float>* bp, const float4* gains) {
  // articulated inertia and bias force at the base: the base body's own, then each leg's in turn
  LegOut<float> sum = base_terms(*bp, B);
  pin(sum);
  const bool corners = corners_may_touch(M, B);
#pragma unroll 1
  for (int leg = 0; leg < 4; ++leg) {
    const LegGains<float> P = load_gains(gains + 2 * leg);
    const float4 a = s.field(kHipTargets + leg);
    const float a3[3] = {a.x, a.y, a.z};
    ParkedWork pw{s.park(leg), 128};
    LegOut<float> o;
    float e[2];
    leg_condense<MS>(M, load_hip(&M.hip[leg]), B, s.leg_state(leg, e), P, a3, pw, o, corners);
    pin(o);
    add_out(sum, o);
  }
  V3<float> d;
  NoFactor none;
  const SV<float> a0 = base_solve_step(M, sum.I, sum.p, B, d, none);
  carry_add(B.p, pe, d);
  pin(B);
#pragma unroll 1
  for (int leg = 0; leg < 4; ++leg) {
    float e[2];
    LegState<float> L = s.leg_state(leg, e);
    LegWork<float> lw;
    unpark_legwork(lw, s.park(leg), 128);
    joint_step(M, a0, lw, L, e);
    s.put_leg_state(leg, L, e);
  }
}

// The final-step error components of one lane's window w from its final state,
// weighted and summed over the eight lanes of the window group (inactive lanes add zero); the
// group's first lane writes them to out (null: nothing is written). Non-finite states count
// into n_bad.
__device__ __forceinline__ void window_result(const WinView& win, int w, bool active, float s13[13],
                                              LegState<float> L[4], float* out, unsigned long long* n_bad) {
  const int W = win.W;
  const float* tgt = win.tgt;
  float sp = 0.f, sq = 0.f, sv = 0.f, sw = 0.f, sj = 0.f, sjd = 0.f;
  bool finite = true;
#pragma unroll
  for (int i = 0; i < 13; ++i) {
    pin(s13[i]);
    const float d = s13[i] - __ldg(tgt + i * W + w);
    finite = finite && isfinite(s13[i]);
    if (i < 3) sp += d * d; else if (i < 7) sq += d * d; else if (i < 10) sv += d * d; else sw += d * d;
  }
#pragma unroll
  for (int leg = 0; leg < 4; ++leg)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float dq = L[leg].q[k] - __ldg(tgt + (13 + 3 * leg + k) * W + w);
      const float dqd = L[leg].qd[k] - __ldg(tgt + (25 + 3 * leg + k) * W + w);
      finite = finite && isfinite(L[leg].q[k]) && isfinite(L[leg].qd[k]);
      sj += dq * dq;
      sjd += dqd * dqd;
    }
  if (active && !finite) atomicAdd(n_bad, 1ull);
  const float wt = active ? __ldg(win.weight + w) : 0.f;
  float comp[SPI_N_COMP] = {sqrtf(sp), sqrtf(sq), sqrtf(sj), sp, sq, sv, sw, sj, sjd};
#pragma unroll
  for (int k = 0; k < SPI_N_COMP; ++k) {
    float c = active ? comp[k] * wt : 0.f;
    pin(c);
    c = group8_sum(c);
    if ((threadIdx.x & 7) == 0 && out) out[k] = c;
  }
}

// Per warp, in 16-byte fields: the lanes' contributions [field][lane] (rows padded to 33), and per
// rollout the base body's constant entries and the sum (rows of 9: conflict-free for the eight
// rollouts of a warp).
struct TeamShare {
  float4 out[8 * 33];
  float4 base[8 * 9];
  float4 sum[8 * 9];
};

// LegOut as eight fields: A 6, B 9, C 6, (3 unused), p 6, (2 unused); p is group 3's own.
__device__ __forceinline__ void pack_out(const LegOut<float>& o, float4 f[8]) {
  const Art<float>& I = o.I;
  f[0] = make_float4(I.A.xx, I.A.yy, I.A.zz, I.A.xy);
  f[1] = make_float4(I.A.xz, I.A.yz, I.B.m[0][0], I.B.m[0][1]);
  f[2] = make_float4(I.B.m[0][2], I.B.m[1][0], I.B.m[1][1], I.B.m[1][2]);
  f[3] = make_float4(I.B.m[2][0], I.B.m[2][1], I.B.m[2][2], I.C.xx);
  f[4] = make_float4(I.C.yy, I.C.zz, I.C.xy, I.C.xz);
  f[5] = make_float4(I.C.yz, 0.f, 0.f, 0.f);
  f[6] = make_float4(o.p.w.x, o.p.w.y, o.p.w.z, o.p.v.x);
  f[7] = make_float4(o.p.v.y, o.p.v.z, 0.f, 0.f);
}
__device__ __forceinline__ LegOut<float> unpack_out(const float4 f[8]) {
  LegOut<float> o;
  Art<float>& I = o.I;
  I.A.xx = f[0].x; I.A.yy = f[0].y; I.A.zz = f[0].z; I.A.xy = f[0].w; I.A.xz = f[1].x; I.A.yz = f[1].y;
  I.B.m[0][0] = f[1].z; I.B.m[0][1] = f[1].w; I.B.m[0][2] = f[2].x;
  I.B.m[1][0] = f[2].y; I.B.m[1][1] = f[2].z; I.B.m[1][2] = f[2].w;
  I.B.m[2][0] = f[3].x; I.B.m[2][1] = f[3].y; I.B.m[2][2] = f[3].z;
  I.C.xx = f[3].w; I.C.yy = f[4].x; I.C.zz = f[4].y; I.C.xy = f[4].z; I.C.xz = f[4].w; I.C.yz = f[5].x;
  o.p.w = v3(f[6].x, f[6].y, f[6].z);
  o.p.v = v3(f[6].w, f[7].x, f[7].y);
  return o;
}
__device__ __forceinline__ float4 add4(float4 a, float4 b) {
  return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

// base (the base body's terms; its constant entries are in share.base already) + FL + FR + RL + RR.
__device__ __forceinline__ LegOut<float> team_sum(TeamShare& share, const LegOut<float>& base, const LegOut<float>& o) {
  const int lane = threadIdx.x & 31, r = lane >> 2, g = lane & 3;
  float4 f[8];
  pack_out(o, f);
#pragma unroll
  for (int i = 0; i < 8; ++i) share.out[i * 33 + lane] = f[i];
  __syncwarp();
  float4 a = share.base[r * 9 + 2 * g], b = share.base[r * 9 + 2 * g + 1];
  if (g == 3) {
    a = make_float4(base.p.w.x, base.p.w.y, base.p.w.z, base.p.v.x);
    b = make_float4(base.p.v.y, base.p.v.z, 0.f, 0.f);
  }
#pragma unroll
  for (int leg = 0; leg < 4; ++leg) {
    a = add4(a, share.out[(2 * g) * 33 + 4 * r + leg]);
    b = add4(b, share.out[(2 * g + 1) * 33 + 4 * r + leg]);
  }
  share.sum[r * 9 + 2 * g] = a;
  share.sum[r * 9 + 2 * g + 1] = b;
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 8; ++i) f[i] = share.sum[r * 9 + i];
  return unpack_out(f);
}

// The legs' constants to shared memory (the lanes of a team index them by leg); the whole CTA.
__device__ __forceinline__ void stage_hip(HipLeg<float> hip[4], const EvalModel& M) {
  if (threadIdx.x < 4 * sizeof(HipLeg<float>) / 16)
    reinterpret_cast<float4*>(hip)[threadIdx.x] = reinterpret_cast<const float4*>(M.hip)[threadIdx.x];
  __syncthreads();
}

// The state of one rollout on a team of lanes: the base on all four, one leg each.
struct TeamRollout {
  BaseState<float> B;
  LegState<float> L;
  V3<float> pe;                // errors carried by B.p and by L.q[1], L.q[2] (carry_add)
  float qe[2];
  BaseParams<float> bp;
  LegGains<float> gains;

  // From the world-frame state x[0 .. 37) at stride `stride` and theta; also stages the base
  // body's constant entries.
  __device__ __forceinline__ void init(const DevModel& M, TeamShare& share, const float* x, size_t stride,
                                       const float* theta) {
    const int lane = threadIdx.x & 31, leg = lane & 3;
    float th[SPI_THETA_DIM];
#pragma unroll
    for (int i = 0; i < SPI_THETA_DIM; ++i) th[i] = __ldg(theta + i);
    bp = base_params<float>(M, th);
    pin(bp.m); pin3(bp.h); pin_s3(bp.Io);
    gains = leg_gains(M, leg_params<float>(th, leg), leg);
    pin(gains);
    float s13[13];
#pragma unroll
    for (int i = 0; i < 13; ++i) s13[i] = x[i * stride];
    base_from_world(B, s13);
    pin(B);
    pe = v3(0.f, 0.f, 0.f);
    qe[0] = qe[1] = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      L.q[k] = x[(13 + 3 * leg + k) * stride];
      L.qd[k] = x[(25 + 3 * leg + k) * stride];
    }
    float4 f[8];
    LegOut<float> own = {};
    own.I = rigid(bp.m, bp.h, bp.Io);
    pack_out(own, f);
    if (leg == 0)
#pragma unroll
      for (int i = 0; i < 8; ++i) share.base[(lane >> 2) * 9 + i] = f[i];
    __syncwarp();
  }

  // One physics substep; hip: the leg's constants, tgt: its joint targets.
  template <int MS>
  __device__ __forceinline__ void substep(const DevModel& M, const HipLeg<float>* hip, const float tgt[3],
                                          TeamShare& share) {
    LegOut<float> base = base_terms(bp, B);
    pin(base);
    LegOut<float> o;
    LegWork<float> W;
    leg_condense<MS>(M, load_hip(hip), B, L, gains, tgt, W, o, corners_may_touch(M, B));
    pin(o);
    pin(W);
    const LegOut<float> sum = team_sum(share, base, o);
    V3<float> d;
    NoFactor none;
    const SV<float> a0 = base_solve_step(M, sum.I, sum.p, B, d, none);
    carry_add(B.p, pe, d);
    pin(B);
    joint_step(M, a0, W, L, qe);
  }
};

}  // namespace spi
