// sensitivity.cu -- per-window state sensitivities d s_H / d theta and Fisher information.
//
// spi_sensitivity: forward-mode (tangent-linear) derivatives of every window's final state
// with respect to K theta slots, for N theta samples. Two ways:
//   * every direction by the dual scalar Df (value + one tangent) through the templated dynamics,
//     one lane quad per (sample, window, direction). Each direction carries the whole trajectory, the
//     legs' condensation and the Cholesky factorisation along: some 4,000 instructions a substep;
//   * the first direction that way, keeping each substep's solve, and the others by tangent.cuh from
//     the kept substeps, one quad per (sample, window, direction) too, 0.46 of the instructions (0.40
//     where a pair's directions share a tape).
// The second runs two chains one after the other, so it takes over where the dual rollouts no longer
// fit the GPU at once (use_tangents).
// With K <= 13 parameters and a 37-dimensional state, K forward tangents give the whole
// Jacobian J_w (37 x K) of each window -- cheaper than 37 reverse (adjoint) sweeps -- and the
// cost gradient follows as dc/dtheta = (dc/ds_H) J_w without checkpointing.
//
// spi_fisher: F_n = sum_w J_w^T diag(q) J_w (FP32 accumulation), log det(F_n + eps I) and
// trace(F_n) in FP64 -- the active-exploration scores (trace is the reference's objective,
// spigym/envs/sysid/active_sysid_openloop.py:402-426; log det the D-optimal one).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "dual.cuh"
#include "engine_impl.h"
#include "kept.cuh"
#include "rollout.cuh"
#include "tangent.cuh"

using namespace spi;

namespace {

__device__ __forceinline__ Df dq_sum(Df x) {
  x.v += __shfl_xor_sync(0xffffffffu, x.v, 1);
  x.d += __shfl_xor_sync(0xffffffffu, x.d, 1);
  x.v += __shfl_xor_sync(0xffffffffu, x.v, 2);
  x.d += __shfl_xor_sync(0xffffffffu, x.d, 2);
  return x;
}
__device__ __forceinline__ void dq_sum_out(LegOut<Df>& o) {
  o.I.A.xx = dq_sum(o.I.A.xx); o.I.A.yy = dq_sum(o.I.A.yy); o.I.A.zz = dq_sum(o.I.A.zz);
  o.I.A.xy = dq_sum(o.I.A.xy); o.I.A.xz = dq_sum(o.I.A.xz); o.I.A.yz = dq_sum(o.I.A.yz);
  o.I.C.xx = dq_sum(o.I.C.xx); o.I.C.yy = dq_sum(o.I.C.yy); o.I.C.zz = dq_sum(o.I.C.zz);
  o.I.C.xy = dq_sum(o.I.C.xy); o.I.C.xz = dq_sum(o.I.C.xz); o.I.C.yz = dq_sum(o.I.C.yz);
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) o.I.B.m[i][j] = dq_sum(o.I.B.m[i][j]);
  o.p.w.x = dq_sum(o.p.w.x); o.p.w.y = dq_sum(o.p.w.y); o.p.w.z = dq_sum(o.p.w.z);
  o.p.v.x = dq_sum(o.p.v.x); o.p.v.y = dq_sum(o.p.v.y); o.p.v.z = dq_sum(o.p.v.z);
}

struct SensArgs {
  int ids[SPI_THETA_DIM];   // the theta slot of each direction
  int K;                 // directions: the columns of J
  long long nw0, nw;     // this launch's (sample, window) pairs
  float* J;              // [N][W][37][K]
  float* xH;             // [N][W][37] or null
  float4* legs;          // kept substeps of the launch's pairs (kept.cuh)
  float4* base;

  __device__ __forceinline__ Kept kept(long long r, int leg) const { return Kept::of(legs, base, (size_t)nw, (size_t)r, leg); }
};

// The work record of the dual rollout that keeps its substeps: also the inverse pivots and the
// contact's branch.
struct DualWork : LegWork<Df> {
  float diag[3], zf, fn, scale;
  __device__ __forceinline__ void put_diag(Df a, Df b, Df c) { diag[0] = a.v; diag[1] = b.v; diag[2] = c.v; }
  __device__ __forceinline__ void put_contact(Df z, const Df* branch) { zf = z.v; fn = branch[0].v; scale = branch[1].v; }
};
__device__ __forceinline__ SV<float> values(const SV<Df>& a) {
  SV<float> r;
  r.w = v3(a.w.x.v, a.w.y.v, a.w.z.v);
  r.v = v3(a.v.x.v, a.v.y.v, a.v.z.v);
  return r;
}
__device__ __forceinline__ BaseState<float> values(const BaseState<Df>& B) {
  BaseState<float> r;
  r.p = v3(B.p.x.v, B.p.y.v, B.p.z.v);
  r.qx = B.qx.v; r.qy = B.qy.v; r.qz = B.qz.v; r.qw = B.qw.v;
  r.nu = values(B.nu);
  return r;
}
__device__ __forceinline__ LegState<float> values(const LegState<Df>& L) {
  LegState<float> r;
#pragma unroll
  for (int k = 0; k < 3; ++k) { r.q[k] = L.q[k].v; r.qd[k] = L.qd[k].v; }
  return r;
}

// KEEP = false: one lane quad per (pair, direction k < K), 8 quads per warp. KEEP = true: direction 0 only, one
// quad per pair, keeping every substep and the final state.
template <bool KEEP>
__global__ void __launch_bounds__(128) sensitivity_kernel(const DevModel* __restrict__ model, WinView win,
                                                          const float* __restrict__ theta,
                                                          const __grid_constant__ SensArgs a) {
  __shared__ DevModel M;
  load_model_smem(&M, model);
  __syncthreads();
  const int lane = threadIdx.x & 31, leg = lane & 3;
  const int per = KEEP ? 1 : a.K;
  const long long total = a.nw * per;
  long long q = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 2;
  const bool active = q < total;
  if (!active) q = total - 1;
  const int k = (int)(q % per);
  const long long r = q / per, nw = a.nw0 + r;
  const int w = (int)(nw % win.W), n = (int)(nw / win.W);
  const int W = win.W, H = win.H;
  const int slot = a.ids[k];

  Df th[SPI_THETA_DIM];
#pragma unroll
  for (int i = 0; i < SPI_THETA_DIM; ++i)
    th[i] = Df(__ldg(theta + (size_t)n * SPI_THETA_DIM + i), i == slot ? 1.f : 0.f);
  const BaseParams<Df> bp = base_params<Df>(M, th);
  const LegParams<Df> lp = leg_params<Df>(th, leg);
  BaseState<Df> B;
  LegState<Df> L;
  {
    Df s13[13];
#pragma unroll
    for (int i = 0; i < 13; ++i) s13[i] = Df(__ldg(win.init + i * W + w));
    base_from_world(B, s13);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      L.q[j] = Df(__ldg(win.init + (13 + 3 * leg + j) * W + w));
      L.qd[j] = Df(__ldg(win.init + (25 + 3 * leg + j) * W + w));
    }
  }
  for (int h = 0; h < H; ++h) {
    const float* ap = win.act + ((size_t)h * W + w) * 12 + 3 * leg;
    Df act[3] = {Df(__ldg(ap)), Df(__ldg(ap + 1)), Df(__ldg(ap + 2))};
    for (int s = 0; s < M.decimation; ++s) {
      if (KEEP) {
        const Kept kept = a.kept(r, leg);
        const int at = h * M.decimation + s;
        keep_state(kept, at, leg, values(B));
        const float nuz = B.nu.v.z.v;
        DualWork lw;
        LegOut<Df> o = phase_a(M, leg, B, L, lp, act, lw);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const SV<float> v = values(lw.Kp[c]);
          const float l = c == 0 ? lw.l10.v : (c == 1 ? lw.l20.v : lw.l21.v);
          __stcs(kept.leg_at(at, 2 * c), make_float4(v.w.x, v.w.y, v.w.z, v.v.x));
          __stcs(kept.leg_at(at, 2 * c + 1), make_float4(v.v.y, v.v.z, lw.y[c].v, l));
        }
        keep_legs(kept, at, lw.diag, values(L), lw.zf, (lw.fn > 0.f ? 1.f : 0.f) + (lw.scale == M.ct ? 2.f : 0.f));
        dq_sum_out(o);
        Art<Df> IA = rigid(bp.m, bp.h, bp.Io);
        add_to(IA, o.I);
        const SV<Df> pA = crf_acc(B.nu, rigid_mul(bp.m, bp.h, bp.Io, B.nu), o.p);
        V3<Df> d;
        Factor6 fac;
        const SV<Df> a0 = base_solve_step(M, IA, pA, B, d, fac);
        B.p = B.p + d;
        keep_solve(kept, at, leg, nuz, values(a0), fac);
        phase_c(M, leg, a0, lw, L);
      } else {
        LegWork<Df> lw;
        LegOut<Df> o = phase_a(M, leg, B, L, lp, act, lw);
        dq_sum_out(o);
        SV<Df> a0 = phase_b(M, bp, o, B);
        phase_c(M, leg, a0, lw, L);
      }
    }
  }
  if (KEEP) {
    const Kept kept = a.kept(r, leg);
    const int at = H * M.decimation;
    const float none[3] = {0.f, 0.f, 0.f};
    keep_state(kept, at, leg, values(B));
    if (leg == 0) *kept.base_at(at, 3) = make_float4(B.nu.v.z.v, 0.f, 0.f, 0.f);
    keep_legs(kept, at, none, values(L));
  }
  if (!active) return;
  Df s13[13];
  base_to_world(B, s13);
  float* Jp = a.J + ((size_t)nw * SPI_STATE_DIM) * a.K + k;
  float* xp = a.xH ? a.xH + (size_t)nw * SPI_STATE_DIM : nullptr;
  if (leg == 0) {
#pragma unroll
    for (int i = 0; i < 13; ++i) {
      Jp[(size_t)i * a.K] = s13[i].d;
      if (xp && k == 0) xp[i] = s13[i].v;
    }
  }
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    Jp[(size_t)(13 + 3 * leg + j) * a.K] = L.q[j].d;
    Jp[(size_t)(25 + 3 * leg + j) * a.K] = L.qd[j].d;
    if (xp && k == 0) {
      xp[13 + 3 * leg + j] = L.q[j].v;
      xp[25 + 3 * leg + j] = L.qd[j].v;
    }
  }
}

constexpr int kKeptFields = 4 * kLegFields + kBaseFields;   // a kept substep of one rollout
constexpr int kTapeFields = 25;   // a leg's tape (24, and one that sets the legs four banks apart)

// What leg_residual_tan reads of a leg's tape, and the joint accelerations.
__device__ __forceinline__ void store_tape(float4* d, const adj::LegTape<float>& t, const float qdd[3]) {
  d[0] = make_float4(t.c[0], t.c[1], t.c[2], t.mimp);
  d[1] = make_float4(t.s[0], t.s[1], t.s[2], t.vf.x);
  d[2] = make_float4(t.vf.y, t.vf.z, qdd[0], qdd[1]);
  const SV<float> v[12] = {t.v0, t.v1, t.v2, t.al0, t.al1, t.al2, t.h0, t.h1, t.h2, t.f0, t.f1, t.f2};
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    const SV<float>&a = v[2 * i], &b = v[2 * i + 1];
    d[3 + 3 * i] = make_float4(a.w.x, a.w.y, a.w.z, a.v.x);
    d[4 + 3 * i] = make_float4(a.v.y, a.v.z, b.w.x, b.w.y);
    d[5 + 3 * i] = make_float4(b.w.z, b.v.x, b.v.y, b.v.z);
  }
  d[21] = make_float4(t.g1.x, t.g1.y, t.g1.z, t.g2.x);
  d[22] = make_float4(t.g2.y, t.g2.z, t.g3.x, t.g3.y);
  d[23] = make_float4(t.g3.z, qdd[2], 0.f, 0.f);
}
__device__ __forceinline__ void load_tape(const float4* d, adj::LegTape<float>& t, float qdd[3]) {
  t.c[0] = d[0].x; t.c[1] = d[0].y; t.c[2] = d[0].z; t.mimp = d[0].w;
  t.s[0] = d[1].x; t.s[1] = d[1].y; t.s[2] = d[1].z;
  t.vf = v3(d[1].w, d[2].x, d[2].y);
  qdd[0] = d[2].z; qdd[1] = d[2].w; qdd[2] = d[23].y;
  SV<float>* const v[12] = {&t.v0, &t.v1, &t.v2, &t.al0, &t.al1, &t.al2, &t.h0, &t.h1, &t.h2, &t.f0, &t.f1, &t.f2};
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    SV<float>&a = *v[2 * i], &b = *v[2 * i + 1];
    const float4 x = d[3 + 3 * i], y = d[4 + 3 * i], z = d[5 + 3 * i];
    a.w = v3(x.x, x.y, x.z); a.v = v3(x.w, y.x, y.y);
    b.w = v3(y.z, y.w, z.x); b.v = v3(z.y, z.z, z.w);
  }
  t.g1 = v3(d[21].x, d[21].y, d[21].z);
  t.g2 = v3(d[21].w, d[22].x, d[22].y);
  t.g3 = v3(d[22].z, d[22].w, d[23].x);
}

// Directions 1 .. K - 1 from the kept substeps, one lane quad per (pair, direction), a pair's directions side by
// side. Bound by its arithmetic at the 8 or 12 warps per SM that its registers leave (0.67, 0.63 instructions a
// cycle; with TAPES the warps wait for the one that forms the next tape). The CTA's pairs (three or four for
// K = 13) have their kept substeps staged through shared memory by asynchronous copies two substeps ahead,
// three buffers in turn; read straight from memory, two warps per scheduler waited for each substep's loads
// twice (1.5 ms at 4096 pairs x 12 directions x H = 20; 1.2 ms so).
//
// TAPES: the part of the residual that a pair's directions share (sines, velocities, accelerations, forces: a
// third of a direction's instructions) is formed once per pair, a substep ahead, one lane per leg, the
// warps taking turns, and read from shared memory. Without its registers three CTAs fit an SM. The
// results are the same to the bit.
template <bool TAPES>
__global__ void __launch_bounds__(128, TAPES ? 3 : 2) tangent_kernel(const DevModel* __restrict__ model, WinView win,
                                                      const float* __restrict__ theta,
                                                      const __grid_constant__ SensArgs a, int stage_pairs) {
  extern __shared__ float4 stage[];               // [3][stage_pairs][kKeptFields]
  float4* const tapes = stage + 3 * stage_pairs * kKeptFields;   // [2][stage_pairs][4][kTapeFields]
  __shared__ DevModel M;
  load_model_smem(&M, model);
  __syncthreads();
  const int lane = threadIdx.x & 31, leg = lane & 3;
  const long long total = a.nw * (a.K - 1);
  const long long q0 = (long long)blockIdx.x * 32;
  long long q = q0 + (threadIdx.x >> 2);
  const bool active = q < total;
  if (!active) q = total - 1;
  const long long first = q0 / (a.K - 1);
  const int pairs = (int)(min(q0 + 31, total - 1) / (a.K - 1) - first) + 1;   // <= stage_pairs
  const int k = 1 + (int)(q % (a.K - 1));
  const long long r = q / (a.K - 1), nw = a.nw0 + r;
  const int W = win.W, H = win.H, w = (int)(nw % W), n = (int)(nw / W);
  const int slot = a.ids[k];
  float th[SPI_THETA_DIM];
#pragma unroll
  for (int i = 0; i < SPI_THETA_DIM; ++i) th[i] = __ldg(theta + (size_t)n * SPI_THETA_DIM + i);
  const BaseParams<float> bp = base_params<float>(M, th);
  const LegParams<float> lp = leg_params<float>(th, leg);
  tng::ParamTan<float> dP;
  tng::base_params_tan(M, th, slot, dP.m, dP.h, dP.Io);
  const int s0 = leg >= 2 ? 9 : 5;
  dP.kps = slot == s0 ? 1.f : 0.f;
  dP.fc = slot == s0 + 1 ? 1.f : 0.f;
  dP.arm = slot == s0 + 2 ? 1.f : 0.f;
  dP.ts = slot == s0 + 3 ? 1.f : 0.f;
  const int last = H * M.decimation;               // the slot of the final state
  auto fetch = [&](int at) {
    if (at <= last)
      for (int i = threadIdx.x; i < pairs * kKeptFields; i += blockDim.x) {
        const int p = i / kKeptFields, f = i - p * kKeptFields;
        const Kept from = a.kept(first + p, f < 4 * kLegFields ? f / kLegFields : 0);
        const float4* src = f < 4 * kLegFields ? from.leg_at(at, f % kLegFields) : from.base_at(at, f - 4 * kLegFields);
        copy_async(stage + ((at % 3) * stage_pairs + p) * kKeptFields + f, src);
      }
    copy_async_commit();
  };
  auto view_of = [&](int at, int p) {
    const float4* f = stage + ((at % 3) * stage_pairs + p) * kKeptFields;
    return KeptView{f + leg * kLegFields, f + 4 * kLegFields};
  };
  auto tape = [&](int at, int p) { return tapes + (((at & 1) * stage_pairs + p) * 4 + leg) * kTapeFields; };
  auto view = [&](int at) { return view_of(at, (int)(r - first)); };
  const int warp = threadIdx.x >> 5;
  // the CTA's tapes of a substep, one lane per leg of a pair, eight pairs a warp; the warps take turns
  auto make_tapes = [&](int at) {
    const int p = ((warp - at) & 3) * 8 + (lane >> 2);
    if (p >= pairs) return;
    const KeptView k = view_of(at, p);
    const BaseState<float> B = k.state();
    const LegState<float> L = k.leg_state();
    const SV<float> a0 = k.accel();
    float qdd[3], none[3] = {0.f, 0.f, 0.f}, res[3];   // (the torques do not enter the tape)
    SV<float> fb;
    adj::LegTape<float> t;
    adj::leg_qdd(k.work(), a0, qdd);
    adj::leg_pose(B, L, t);
    adj::leg_residual<kMotorRuntime>(M, leg, B, L, lp, none, a0, qdd, t, res, fb);
    store_tape(tape(at, p), t, qdd);
  };
  auto arrive = [&] {
    copy_async_wait<0>();
    __syncthreads();
  };
  fetch(0);
  fetch(1);
  arrive();
  if (TAPES) {
    make_tapes(0);
    __syncthreads();
  }
  BaseState<float> B0 = view(0).state();
  tng::BaseTan<float> dB = tng::zero_base_tan<float>();
  tng::LegTan<float> dL = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
  for (int h = 0; h < H; ++h) {
    float tgt[3];
#pragma unroll
    for (int j = 0; j < 3; ++j)
      tgt[j] = joint_target(M, j, leg, __ldg(win.act + ((size_t)h * W + w) * 12 + 3 * leg + j));
    for (int s = 0; s < M.decimation; ++s) {
      const int at = h * M.decimation + s;
      if (at > 0) arrive();                        // slot at + 1 and tape at are here, at - 1's are free
      fetch(at + 2);
      if (TAPES && at + 1 < last) make_tapes(at + 1);
      const KeptView now = view(at);
      const LegState<float> L = now.leg_state();
      const float4 c = now.legf(8);
      const int branch = (int)c.z;
      const tng::ContactBranch br = {(branch & 1) != 0, (branch & 2) != 0};
      const SV<float> a0 = now.accel();
      float qdd[3], dr[3], z[3], dqdd[3];
      SV<float> x;
      {
        adj::LegTape<float> t;
        if (TAPES) {
          load_tape(tape(at, (int)(r - first)), t, qdd);
        } else {
          float res[3];
          SV<float> fb;
          adj::leg_qdd(now.work(), a0, qdd);
          adj::leg_pose(B0, L, t);
          adj::leg_residual<kMotorRuntime>(M, leg, B0, L, lp, tgt, a0, qdd, t, res, fb);
        }
        tng::leg_residual_tan(M, leg, B0, L, lp, tgt, qdd, t, c.y, br, dB, dL, dP, dr, x);
      }
      if (corners_may_touch(M, B0)) {
#pragma unroll
        for (int j = 0; j < 2; ++j)
          adj::add_sv(x, tng::corner_residual_tan(M, B0, lc_corner<float>(M.legc[leg], j), a0, dB));
      }
      // M' da = -dr
      const float lam[3] = {-dr[0], -dr[1], -dr[2]};
      const adj::SolveWork<float> sw = now.work();
      adj::add_sv(x, adj::leg_solve_down(sw, lam, z));
      qsum3(x.w);
      qsum3(x.v);
      adj::add_sv(x, tng::base_residual_tan(bp, B0, a0, dB, dP));
      const SV<float> da0 = now.factor().solve(adj::sub_sv(adj::zsv<float>(), x));
      adj::leg_solve_up(sw, z, da0, dqdd);
      const BaseState<float> B1 = view(at + 1).state();
      tng::base_integrate_tan(M, B0, B1, da0, dB);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        dL.qd[j] = dL.qd[j] + M.dt * dqdd[j];
        dL.q[j] = dL.q[j] + M.dt * dL.qd[j];
      }
      B0 = B1;
    }
  }
  if (!active) return;
  float s13[13];
  tng::base_to_world_tan(B0, dB, s13);
  float* Jp = a.J + ((size_t)nw * SPI_STATE_DIM) * a.K + k;
  if (leg == 0) {
#pragma unroll
    for (int i = 0; i < 13; ++i) Jp[(size_t)i * a.K] = s13[i];
  }
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    Jp[(size_t)(13 + 3 * leg + j) * a.K] = dL.q[j];
    Jp[(size_t)(25 + 3 * leg + j) * a.K] = dL.qd[j];
  }
}

// Whether the directions past the first go by tangents: three directions or more whose dual rollouts would
// take more than `waves` times the warps that fit the GPU at once (two CTAs of 255 registers a thread per
// SM). The first direction's chain comes before the others', so below two waves the dual rollouts are done
// first, and with two directions it does not come back (H = 20, 152 SMs, dual against tangents):
//   1100 pairs x 13   0.80 / 0.85 ms      1530 x 13   1.16 / 0.86 ms      4096 x 13   2.33 / 1.55 ms
//   4900 pairs x 3    0.79 / 0.96 ms      6600 x 3    1.15 / 1.03 ms     10000 x 2    1.13 / 1.35 ms
// Batches follow one another, each with a last wave of its own, so that several of them ask for more each. Five
// batches at 2.2, 3.0 and 3.7 waves: H = 200, K = 3, 4, 5: 45.8 / 50.5, 60.2 / 60.1, 74.2 / 58.0 ms; H = 400, K = 6, 8,
// 10: 91.9 / 92.4, 121 / 112, 149 / 131. Four waves, at which none of them loses.
constexpr int kDualWaves = 2;
bool use_tangents(long long pairs, int K, int sms, int waves) {
  return K >= 3 && pairs * K > (long long)waves * 2 * 32 * sms;
}

// A CTA's staged pairs (32 consecutive quads touch so many at most) and its dynamic shared memory, bytes.
int stage_pairs_of(int K) { return 31 / (K - 1) + 2; }
int tangent_smem(int K, bool tapes) {
  return stage_pairs_of(K) * (3 * kKeptFields + (tapes ? 8 * kTapeFields : 0)) * (int)sizeof(float4);
}

// Whether the tangents of a pair share one tape: with four or more to share it, and over two waves of the two
// CTAs per SM that fit otherwise (H = 20, 152 SMs, whole call, own tapes against shared ones):
//   4096 pairs x 13   1.67 / 1.55 ms      1650 x 13   0.98 / 0.94 ms      1530 x 13   0.86 / 0.94 ms
//   8192 pairs x 5    1.40 / 1.40 ms      8192 x 4    1.23 / 1.28 ms      4096 x 5    0.96 / 1.05 ms
bool use_tapes(long long pairs, int K, int sms) {
  return K >= 5 && pairs * (K - 1) > (long long)2 * 2 * 32 * sms;
}

// ---------------------------------------------------------------------------
// Fisher information: F[n] = sum_w J^T diag(q) J, log det(F + eps I) and trace(F), two samples a CTA.
//
// J is read once, coalesced, kFisherRows rows at a time (the next rows are on their way in registers while
// these are summed), into shared memory in the layout the accumulation reads; the sums run from there
// in row order, as one chain per entry (FP32) or per 8-column tile of the m16n8k16 product (tensor
// cores), so the staging does not show in a result. The scores follow in the same launch, both
// samples on one warp (a sample has 13 rows at most, and an FP64 instruction takes as long for one
// lane as for 32). 512 samples x 8 windows x 13 parameters, BF16: 115 -> 16.5 us. For many samples the
// scores, and of few windows the sums too, come from kernels with less fixed work a sample (many_samples,
// few_rows below); a sample's results are the same to the bit by each.
// ---------------------------------------------------------------------------
constexpr int kFisherRows = 128;                 // rows of J staged at a time (a multiple of 16)
constexpr int kFisherPitch = kFisherRows / 2 + 4;   // words per parameter of the BF16 tile; 4 mod 32: conflict-free
constexpr int kFisherThreads = 128;              // per sample
constexpr int kFisherPer = kFisherRows * SPI_THETA_DIM / kFisherThreads;   // elements a thread stages

// log det(F + eps I) by an FP64 L D L^T and trace(F), row i on lane i of a half-warp. A column's pivot and
// entries go round by shuffles; each entry's subtractions run in the order k = 0 .. j - 1. logdet / trace
// null: not written.
__device__ __forceinline__ void fisher_scores(const float* F, int K, double eps, double* logdet, double* trace) {
  const int i = threadIdx.x & 15;
  double row[SPI_THETA_DIM];
#pragma unroll
  for (int j = 0; j < SPI_THETA_DIM; ++j)
    row[j] = i < K && j < K ? (double)F[i * K + j] + (j == i ? eps : 0.0) : 0.0;
  const double diag = i < K ? (double)F[i * K + i] : 0.0;
  double pivot = 1.0, tr = 0.0;
  bool ok = true;
#pragma unroll
  for (int j = 0; j < SPI_THETA_DIM; ++j) {
    if (j < K) {                                  // uniform
      const double t = __shfl_sync(0xffffffffu, diag, j, 16);
      if (ok) tr += t;
      const double d = __shfl_sync(0xffffffffu, row[j], j, 16);
      ok = ok && d > 0.0;
      if (i == j) pivot = d;
      const double l = row[j] * (1.0 / d);
#pragma unroll
      for (int k = j + 1; k < SPI_THETA_DIM; ++k)
        if (k < K) row[k] = fma(-l, __shfl_sync(0xffffffffu, row[j], k, 16), row[k]);
    }
  }
  const double lg = log(pivot);
  double ld = 0.0;
  for (int j = 0; j < K; ++j) ld += __shfl_sync(0xffffffffu, lg, j, 16);
  if (i == 0) {
    if (logdet) *logdet = ok ? ld : -INFINITY;
    if (trace) *trace = tr;
  }
}

// The same, in the same operations, from F in memory with one sample a thread, for many samples: a warp's FP64
// instruction then serves 32 samples (fisher_scores: two), but a sample is one thread's chain. The lower
// triangle is in registers.
__global__ void __launch_bounds__(32) fisher_scores_kernel(const float* __restrict__ F, int N, int K, double eps,
                                                           double* __restrict__ logdet, double* __restrict__ trace) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  const float* f = F + (size_t)n * K * K;
  double A[SPI_THETA_DIM][SPI_THETA_DIM];
#pragma unroll
  for (int i = 0; i < SPI_THETA_DIM; ++i)
#pragma unroll
    for (int j = 0; j <= i; ++j) A[i][j] = i < K ? (double)f[i * K + j] + (j == i ? eps : 0.0) : 0.0;
  double ld = 0.0, tr = 0.0;
  bool ok = true;
#pragma unroll
  for (int j = 0; j < SPI_THETA_DIM; ++j) {
    if (j >= K) break;                            // uniform
    if (ok) tr += (double)f[j * K + j];
    const double d = A[j][j];
    ok = ok && d > 0.0;
    ld += log(d);
    const double inv = 1.0 / d;
#pragma unroll
    for (int i = j + 1; i < SPI_THETA_DIM; ++i)
      if (i < K) {
        const double l = A[i][j] * inv;
#pragma unroll
        for (int k = j + 1; k <= i; ++k) A[i][k] = fma(-l, A[k][j], A[i][k]);
      }
  }
  if (logdet) logdet[n] = ok ? ld : -INFINITY;
  if (trace) trace[n] = tr;
}
// TC = false: FP32 on the CUDA cores, one entry (p, r >= p) a thread: acc += (q J_p) J_r over the rows.
// TC = true: BF16 operands (Q^1/2 J), FP32 accumulation, mma.sync m16n8k16 by one warp: A = (Q^1/2 J)^T
// as a 16 x 16 tile, B = Q^1/2 J as two 16 x 8 tiles (the same registers: A's row groups are B's columns).
// Rows past W * 37 and parameters past K are zero. (13 parameters fill a fifth of the smallest tcgen05
// tile, M = 64; the product is a few microseconds of one warp here.)
template <bool TC>
__global__ void __launch_bounds__(2 * kFisherThreads) fisher_kernel(const float* __restrict__ J, int N, int W, int K,
                                                                    const float* __restrict__ q, double eps,
                                                                    float* __restrict__ F, double* __restrict__ logdet,
                                                                    double* __restrict__ trace) {
  constexpr int kWords = TC ? 16 * kFisherPitch : 2 * kFisherRows * SPI_THETA_DIM;
  __shared__ __align__(16) unsigned tiles[2][kWords];
  __shared__ float s_q[SPI_STATE_DIM];
  __shared__ float s_F[2][SPI_THETA_DIM * SPI_THETA_DIM];
  const int half = threadIdx.x / kFisherThreads, tid = threadIdx.x % kFisherThreads;
  const int lane = tid & 31, g = lane >> 2, t = lane & 3;
  const bool live = (int)(2 * blockIdx.x + half) < N;
  const int n = live ? 2 * blockIdx.x + half : N - 1;          // the odd sample out runs a copy of the last
  unsigned* tile = tiles[half];
  const int rows = W * SPI_STATE_DIM;
  const float* Jn = J + (size_t)n * rows * K;
  if (threadIdx.x < SPI_STATE_DIM) s_q[tid] = q ? (TC ? sqrtf(q[tid]) : q[tid]) : 1.f;
  if (TC)
    for (int i = tid; i < kWords; i += kFisherThreads) tile[i] = 0u;
  // this thread's entry of the FP32 sums
  const int nent = K * (K + 1) / 2;
  int ep = 0, er = tid;
  while (ep < K && er >= K - ep) { er -= K - ep; ++ep; }
  er += ep;
  const unsigned inv_K = 65536u / K + 1;                       // i / K for i < kFisherRows * 13
  float acc = 0.f, c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};
  float next[kFisherPer];
#pragma unroll
  for (int e = 0; e < kFisherPer; ++e) {
    const int i = e * kFisherThreads + tid;
    next[e] = i < min(kFisherRows, rows) * K ? __ldg(Jn + i) : 0.f;
  }
  for (int r0 = 0; r0 < rows; r0 += kFisherRows) {
    const int m = min(kFisherRows, rows - r0), ahead = min(kFisherRows, rows - r0 - kFisherRows) * K;
    __syncthreads();                              // the tile is free (and, at first, s_q and the zeros are set)
#pragma unroll
    for (int e = 0; e < kFisherPer; ++e) {
      const int i = e * kFisherThreads + tid;
      if (i < m * K) {
        const int r = (int)((unsigned)i * inv_K >> 16), p = i - r * K;
        const float v = next[e], w = s_q[(r0 + r) % SPI_STATE_DIM];
        if (TC) {
          reinterpret_cast<__nv_bfloat16*>(tile)[p * 2 * kFisherPitch + r] = __float2bfloat16_rn(w * v);
        } else {
          reinterpret_cast<float*>(tile)[i] = w * v;
          reinterpret_cast<float*>(tile)[kFisherRows * SPI_THETA_DIM + i] = v;
        }
      }
      next[e] = i < ahead ? __ldg(Jn + (size_t)(r0 + kFisherRows) * K + i) : 0.f;
    }
    if (TC && m < kFisherRows)                    // the rows up to the next multiple of 16 are zero
      for (int i = tid; i < 16 * 16; i += kFisherThreads) {
        const int p = i >> 4, r = m + (i & 15);
        if (r < ((m + 15) & ~15)) reinterpret_cast<__nv_bfloat16*>(tile)[p * 2 * kFisherPitch + r] = __float2bfloat16_rn(0.f);
      }
    __syncthreads();
    if (TC) {
      if (tid < 32)
        for (int k0 = 0; k0 < m; k0 += 16) {
          // (rows k0 + 2t, 2t + 1) and (k0 + 2t + 8, 2t + 9) of parameters g and g + 8
          const unsigned* u = tile + g * kFisherPitch + k0 / 2 + t;
          const unsigned* v = u + 8 * kFisherPitch;
          const unsigned a0 = u[0], a1 = v[0], a2 = u[4], a3 = v[4];
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) {
            float* c = nt ? c1 : c0;
            const unsigned b0 = nt ? a1 : a0, b1 = nt ? a3 : a2;
            asm volatile(
                "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                "{%0, %1, %2, %3};\n"
                : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
          }
        }
    } else if (tid < nent) {
      const float* x = reinterpret_cast<const float*>(tile) + ep;
      const float* y = reinterpret_cast<const float*>(tile) + kFisherRows * SPI_THETA_DIM + er;
#pragma unroll 16
      for (int r = 0; r < m; ++r) acc = fmaf(x[r * K], y[r * K], acc);
    }
  }
  float* Fs = s_F[half];
  if (TC) {
    // D fragment: rows g and g + 8, cols 2t and 2t + 1 of each n-tile
    if (tid < 32)
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = g + (e >= 2 ? 8 : 0), j = 8 * nt + 2 * t + (e & 1);
          if (i < K && j < K) Fs[i * K + j] = (nt ? c1 : c0)[e];
        }
  } else if (tid < nent) {
    Fs[ep * K + er] = acc;
    Fs[er * K + ep] = acc;
  }
  __syncthreads();
  if (live)
    for (int i = tid; i < K * K; i += kFisherThreads) F[(size_t)n * K * K + i] = Fs[i];
  if (threadIdx.x < 32 && (logdet || trace)) {
    const int h = threadIdx.x >> 4, s = 2 * blockIdx.x + h;
    fisher_scores(s_F[h], K, eps, logdet && s < N ? logdet + s : nullptr, trace && s < N ? trace + s : nullptr);
  }
}

// The sums of fisher_kernel, in its order, for many samples of few rows: one warp a sample, straight from memory. Staging a
// CTA's tile takes the same instructions however few rows there are.
__device__ __forceinline__ unsigned jq_pair(const float* Jn, const float* q, int rows, int K, int r, int p) {
  float v[2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
    v[i] = r + i < rows && p < K ? (q ? sqrtf(q[(r + i) % SPI_STATE_DIM]) : 1.f) * Jn[(size_t)(r + i) * K + p] : 0.f;
  const __nv_bfloat162 b = __floats2bfloat162_rn(v[0], v[1]);
  return *reinterpret_cast<const unsigned*>(&b);
}
template <bool TC>
__global__ void __launch_bounds__(128) fisher_few_rows_kernel(const float* __restrict__ J, int N, int W, int K,
                                                              const float* __restrict__ q, float* __restrict__ F) {
  const int n = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (n >= N) return;                             // uniform per warp
  const int lane = threadIdx.x & 31, rows = W * SPI_STATE_DIM;
  const float* Jn = J + (size_t)n * rows * K;
  float* Fn = F + (size_t)n * K * K;
  if (TC) {
    const int g = lane >> 2, t = lane & 3;
    float c[2][4] = {};
    for (int k0 = 0; k0 < rows; k0 += 16) {
      const int r = k0 + 2 * t;
      const unsigned a0 = jq_pair(Jn, q, rows, K, r, g), a1 = jq_pair(Jn, q, rows, K, r, g + 8),
                     a2 = jq_pair(Jn, q, rows, K, r + 8, g), a3 = jq_pair(Jn, q, rows, K, r + 8, g + 8);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
        asm volatile(
            "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
            "{%0, %1, %2, %3};\n"
            : "+f"(c[nt][0]), "+f"(c[nt][1]), "+f"(c[nt][2]), "+f"(c[nt][3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(nt ? a1 : a0), "r"(nt ? a3 : a2));
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = g + (e >= 2 ? 8 : 0), j = 8 * nt + 2 * t + (e & 1);
        if (i < K && j < K) Fn[i * K + j] = c[nt][e];
      }
  } else {
    for (int e = lane; e < K * (K + 1) / 2; e += 32) {
      int p = 0, r = e;
      while (r >= K - p) { r -= K - p; ++p; }
      r += p;
      float acc = 0.f;
      for (const float* Jw = Jn; Jw < Jn + rows * K; Jw += SPI_STATE_DIM * K) {
#pragma unroll
        for (int i = 0; i < SPI_STATE_DIM; ++i)
          acc = fmaf((q ? __ldg(q + i) : 1.f) * __ldg(Jw + i * K + p), __ldg(Jw + i * K + r), acc);
      }
      Fn[p * K + r] = acc;
      Fn[r * K + p] = acc;
    }
  }
}

// Whether the scores come in a launch of their own: a sample's take one chain's length then (6 us at K = 1, 38 at
// K = 13), and up to some number of samples the half-warps are done first; FP32 sums of more windows
// hide more of them. us a call, scores in the sums' launch / apart (sums by the better kernel):
//   tensor cores  4096 x 1 x 13  60 / 52    4096 x 8 x 13  76 / 74    3000 x 8 x 8  45 / 46    50000 x 1 x 13  602 / 216
//   FP32          4096 x 1 x 5   25 / 25    6000 x 1 x 13  60 / 62    8192 x 8 x 8  89 / 91    50000 x 1 x 5   222 / 99
bool many_samples(int N, int W, int K, bool tc) {
  return tc ? N > 1700 + 180 * K : (long long)N * 8 > (3000LL + 300 * K) * (8 + W);
}
// Whether the sums of many samples are by fisher_few_rows_kernel (us a call, staged / this one):
//   tensor cores  16384 x 1 x 13  93 / 66    16384 x 4 x 5   82 / 62    16384 x 4 x 13  127 / 126    16384 x 8 x 13  160 / 172
//   FP32          16384 x 1 x 1   38 / 21    16384 x 2 x 5   58 / 50    16384 x 1 x 13   93 / 87     50000 x 4 x 5   233 / 288
bool few_rows(int W, int K, bool tc) { return tc ? W <= 4 : W * K <= 10; }

}  // namespace

cudaError_t spi::sensitivity_prepare() {
  int own = 0, shared = 0;
  for (int K = 3; K <= SPI_THETA_DIM; ++K) {
    own = std::max(own, tangent_smem(K, false));
    shared = std::max(shared, tangent_smem(K, true));
  }
  const cudaError_t ce = cudaFuncSetAttribute(tangent_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, own);
  if (ce != cudaSuccess) return ce;
  return cudaFuncSetAttribute(tangent_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, shared);
}

extern "C" {

int spi_sensitivity(spi_engine* e, const float* theta, int N, const int32_t* param_ids, int K, float* J, float* xH) {
  if (!e || !theta || !param_ids || !J) return set_error(SPI_EINVAL, "spi_sensitivity: null argument");
  if (e->W <= 0) return set_error(SPI_ESTATE, "spi_sensitivity before spi_load_windows");
  if (N <= 0 || K < 1 || K > SPI_THETA_DIM) return set_error(SPI_EINVAL, "spi_sensitivity: N=%d K=%d", N, K);
  for (int k = 0; k < K; ++k)
    if (param_ids[k] < 0 || param_ids[k] >= SPI_THETA_DIM)
      return set_error(SPI_EINVAL, "spi_sensitivity: param_ids[%d]=%d", k, param_ids[k]);
  const WinView win{e->init.f(), e->act.f(), e->tgt.f(), e->weight.f(), e->W, e->H};
  SensArgs a{};
  for (int k = 0; k < K; ++k) a.ids[k] = param_ids[k];
  a.K = K;
  a.J = J;
  a.xH = xH;
  const long long all = (long long)N * e->W;
  const size_t slots = (size_t)e->H * e->host_model.decimation + 1;
  // Batches of equal size within the engine's limit. A capture keeps to the dual rollouts, which need no memory of
  // the engine's: a graph would go on using what a later call may replace.
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  const bool may = cudaStreamIsCapturing(e->stream, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone;
  long long batch = all;
  bool split = false;
  e->sens_limit.begin_call();
  while (may && !split) {
    const long long most = std::max(1LL, (long long)(e->sens_limit.bytes / (slots * kKeptBytes)));
    const long long batches = (all + most - 1) / most;
    batch = (all + batches - 1) / batches;
    if (!use_tangents(batch, K, e->sms, batches > 1 ? 2 * kDualWaves : kDualWaves)) break;
    const size_t need = slots * batch * kKeptBytes;
    split = e->sens_kept.reserve(need) == SPI_OK;
    if (!split) e->sens_limit.refused(need);
  }
  if (!split) batch = all;
  // The results are the caller's and the directions' own rollouts share nothing, so calls on several streams
  // (spi_set_stream) may overlap; the kept substeps are the engine's, and a call on another stream waits for them.
  if (split) {
    cudaError_t ce = e->sens_done ? cudaStreamWaitEvent(e->stream, e->sens_done, 0)
                                  : cudaEventCreateWithFlags(&e->sens_done, cudaEventDisableTiming);
    if (ce != cudaSuccess) return cuda_error(ce, "spi_sensitivity: order of the calls");
  }
  const bool tapes = use_tapes(batch, K, e->sms);
  const auto tangents = tapes ? tangent_kernel<true> : tangent_kernel<false>;
  for (long long r0 = 0; r0 < all; r0 += batch) {
    a.nw0 = r0;
    a.nw = std::min(batch, all - r0);
    if (split) {
      a.legs = (float4*)e->sens_kept.p;
      a.base = a.legs + slots * kLegFields * 4 * a.nw;
      sensitivity_kernel<true><<<blocks_for(a.nw, 32), 128, 0, e->stream>>>(e->d_model, win, theta, a);
      tangents<<<blocks_for(a.nw * (K - 1), 32), 128, tangent_smem(K, tapes), e->stream>>>(e->d_model, win, theta, a,
                                                                                         stage_pairs_of(K));
    } else {
      sensitivity_kernel<false><<<blocks_for(a.nw * K, 32), 128, 0, e->stream>>>(e->d_model, win, theta, a);
    }
  }
  cudaError_t ce = cudaGetLastError();
  if (ce == cudaSuccess && split) ce = cudaEventRecord(e->sens_done, e->stream);
  return ce == cudaSuccess ? SPI_OK : cuda_error(ce, "spi_sensitivity: launch");
}

int spi_fisher(const float* J, int N, int W, int K, const float* state_weight, double eps, float* F, double* logdet,
               double* trace, void* stream) {
  return spi_fisher_ex(J, N, W, K, state_weight, eps, 0, F, logdet, trace, stream);
}

int spi_fisher_ex(const float* J, int N, int W, int K, const float* state_weight, double eps, int tensor_cores,
                  float* F, double* logdet, double* trace, void* stream) {
  if (!J || !F || N <= 0 || W <= 0 || K < 1 || K > SPI_THETA_DIM)
    return set_error(SPI_EINVAL, "spi_fisher: bad argument");
  cudaStream_t s = (cudaStream_t)stream;
  const bool scores = logdet || trace, many = many_samples(N, W, K, tensor_cores != 0);
  if (many && few_rows(W, K, tensor_cores != 0)) {
    const auto kernel = tensor_cores ? fisher_few_rows_kernel<true> : fisher_few_rows_kernel<false>;
    kernel<<<blocks_for(N, 4), 128, 0, s>>>(J, N, W, K, state_weight, F);
  } else {
    const auto kernel = tensor_cores ? fisher_kernel<true> : fisher_kernel<false>;
    kernel<<<blocks_for(N, 2), 2 * kFisherThreads, 0, s>>>(J, N, W, K, state_weight, eps, F, many ? nullptr : logdet,
                                                          many ? nullptr : trace);
  }
  if (many && scores) fisher_scores_kernel<<<blocks_for(N, 32), 32, 0, s>>>(F, N, K, eps, logdet, trace);
  cudaError_t ce = cudaGetLastError();
  return ce == cudaSuccess ? SPI_OK : cuda_error(ce, "spi_fisher");
}

}  // extern "C"
