// adjoint.cu -- spi_adjoint: cost and d cost / d theta of every theta sample by the hand-written
// reverse sweep of the rollout (adjoint.cuh).
//
// Layout: the quad layout of rollout.cuh (CTAs of 128 threads; four lanes per rollout, one leg
// each; one warp = one theta sample x 8 consecutive windows). Per rollout:
//   1. adjoint_forward_kernel runs the control steps and keeps, before every physics substep, the
//      state and what the substep's equations of motion were solved with: each leg's factorisation
//      (L, D^-1, K'), y, the base's Cholesky factor and acceleration;
//   2. adjoint_reverse_kernel forms the final state's cost and its adjoint (the engine's cost mode
//      and weights) and runs the substep adjoints backwards over the kept substeps; the theta
//      adjoint accumulates on the way. Nothing of the forward pass is computed again;
//   3. the window-weighted costs and theta adjoints of the warp's 8 windows are summed (fixed
//      order) into one partial per (theta, window group); adjoint_finalize sums a theta's partials
//      in group order and divides by the window normaliser, as the cost of spi_run does.
// The kept substeps are 736 bytes each per rollout, written and read once in 16-byte fields, a warp's
// accesses contiguous. They take 4 GB at most (ScratchLimit): (theta, group) pairs go through in batches, and a
// horizon over kSegSteps control steps in segments from checkpoints of the state (the segments'
// forward passes run again, last segment first, the adjoint carried in memory).
#include <cuda_runtime.h>

#include <algorithm>

#include "adjoint.cuh"
#include "engine_impl.h"
#include "kept.cuh"
#include "rollout.cuh"

using namespace spi;

namespace {

constexpr int kSegSteps = 50;                       // control steps between checkpoints
constexpr size_t kPairBytes = 8 * kKeptBytes;       // a warp's eight rollouts', per substep

// Phase A's work record to its parking slot (for phase C) and to the kept substep.
struct KeptWork {
  ParkedWork park;
  float4* kept;
  size_t stride;
  float diag[3];
  __device__ __forceinline__ void put_col(int k, const SV<float>& v, float yk, float lk) {
    park.put_col(k, v, yk, lk);
    __stcs(kept + 2 * k * stride, make_float4(v.w.x, v.w.y, v.w.z, v.v.x));
    __stcs(kept + (2 * k + 1) * stride, make_float4(v.v.y, v.v.z, yk, lk));
  }
  __device__ __forceinline__ void put_diag(float a, float b, float c) { diag[0] = a; diag[1] = b; diag[2] = c; }
};

// substep (rollout.cuh), keeping the state it starts from and its factorisations in `slot`.
__device__ __forceinline__ void substep_kept(const DevModel& M, int leg, BaseState<float>& B, LegState<float>& L,
                                             const BaseParams<float>& bp, const LegParams<float>& lp,
                                             const float act[3], const Kept& k, int slot) {
  __shared__ float4 lw_smem[kParkVec * 128];
  KeptWork kw{ParkedWork{lw_smem + threadIdx.x, 128}, k.leg_at(slot, 0), k.leg_field, {0.f, 0.f, 0.f}};
  keep_state(k, slot, leg, B);
  const float nuz = B.nu.v.z;
  LegOut<float> o = phase_a(M, leg, B, L, lp, act, kw);
  keep_legs(k, slot, kw.diag, L);
  qsum_out(o);
  Art<float> IA = rigid(bp.m, bp.h, bp.Io);
  add_to(IA, o.I);
  const SV<float> pA = crf_acc(B.nu, rigid_mul(bp.m, bp.h, bp.Io, B.nu), o.p);
  V3<float> d;
  Factor6 fac;
  const SV<float> a0 = base_solve_step(M, IA, pA, B, d, fac);
  B.p = B.p + d;
  keep_solve(k, slot, leg, nuz, a0, fac);
  LegWork<float> lw;
  unpark_legwork(lw, lw_smem + threadIdx.x, 128);
  phase_c(M, leg, a0, lw, L);
}

__device__ __forceinline__ void qsum_sv(SV<float>& s) { qsum3(s.w); qsum3(s.v); }

// One substep's adjoint on a lane quad (lane = leg): lam / lq / lqd hold the adjoint of the
// state after the substep (its base: B1) on entry and of B0 / L0 on exit; gth accumulates the theta
// adjoint (the lane's leg-group slots; lane 0 also the base slots). W, fac, a0: the substep's kept
// factorisations and base acceleration.
__device__ __forceinline__ void substep_adjoint(const DevModel& M, int leg, const BaseState<float>& B0,
                                                const LegState<float>& L0, const BaseState<float>& B1,
                                                const adj::SolveWork<float>& W, const Factor6& fac, const SV<float>& a0,
                                                const BaseParams<float>& bp, const LegParams<float>& lp, const float* th,
                                                const float act[3], adj::BaseAdj<float>& lam, float lq[3], float lqd[3],
                                                float gth[13]) {
  adj::LegTape<float> t;
  adj::leg_pose(B0, L0, t);
  float qdd[3];
  adj::leg_qdd(W, a0, qdd);
  // integrator backwards (the base part is the same on the four lanes)
  adj::BaseAdj<float> lam0;
  SV<float> a0b;
  M3<float> R0b = adj::zm3<float>();
  adj::base_integrate_bar(M, B0, B1, lam, lam0, a0b, R0b);
  float qb0[3], qdb0[3], qddb[3];
  adj::leg_integrate_bar(M, lq, lqd, qb0, qdb0, qddb);
  // mu = M'^-1 (a0b; qddb)
  float z[3];
  SV<float> kz = adj::leg_solve_down(W, qddb, z);
  qsum_sv(kz);
  const SV<float> mub = fac.solve(adj::sub_sv(a0b, kz));
  float mu[3];
  adj::leg_solve_up(W, z, mub, mu);
  // the residual backwards with the seed mu
  float tgt[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) tgt[k] = joint_target(M, k, leg, act[k]);
  float r[3];
  SV<float> fb;
  adj::leg_residual<kMotorRuntime>(M, leg, B0, L0, lp, tgt, a0, qdd, t, r, fb);
  adj::BaseBar<float> bb = adj::zero_base_bar<float>();
  float qb[3] = {0.f, 0.f, 0.f}, qdb[3] = {0.f, 0.f, 0.f};
  adj::LegParamBar<float> pb = {0.f, 0.f, 0.f, 0.f};
  adj::leg_residual_bar<kMotorRuntime>(M, leg, B0, L0, lp, tgt, a0, qdd, t, mu, mub, bb, qb, qdb, pb);
  if (corners_may_touch(M, B0)) {
#pragma unroll
    for (int j = 0; j < 2; ++j) adj::corner_residual_bar(M, B0, lc_corner<float>(M.legc[leg], j), a0, mub, bb);
  }
  if (leg == 0) {
    float mb = 0.f;
    V3<float> hb = adj::z3<float>();
    S3<float> Iob;
    Iob.xx = Iob.yy = Iob.zz = Iob.xy = Iob.xz = Iob.yz = 0.f;
    adj::base_residual_bar(bp, B0, a0, mub, bb, mb, hb, Iob);
    float gb[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
    adj::base_params_bar(M, th, mb, hb, Iob, gb);
#pragma unroll
    for (int i = 0; i < 5; ++i) gth[i] -= gb[i];
  }
  // the base adjoints of the four legs (and the base's own terms) summed
  bb.pz = qsum(bb.pz);
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) bb.R.m[i][j] = qsum(bb.R.m[i][j]);
  qsum_sv(bb.nu);
  lam0.p.z -= bb.pz;
  lam0.nu = adj::sub_sv(lam0.nu, bb.nu);
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) R0b.m[i][j] -= bb.R.m[i][j];
  adj::quat_to_R_bar(B0.qx, B0.qy, B0.qz, B0.qw, R0b, lam0.qx, lam0.qy, lam0.qz, lam0.qw);
  lam = lam0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    lq[k] = qb0[k] - qb[k];
    lqd[k] = qdb0[k] - qdb[k];
  }
  const float pg[4] = {pb.kps, pb.fc, pb.arm, pb.ts};
#pragma unroll
  for (int i = 0; i < 4; ++i) {   // selects, not a run-time index: keeps gth in registers
    gth[5 + i] -= leg < 2 ? pg[i] : 0.f;
    gth[9 + i] -= leg < 2 ? 0.f : pg[i];
  }
}

struct AdjArgs {
  WinView win;
  const float* theta;
  int G, mode;
  float w[6];          // squared-error block weights (mode 1)
  long long pair0, pairs;   // this batch: (theta, group) pairs pair0 .. pair0 + pairs
  int h0, h1, H;       // this segment's control steps; the horizon
  float4* legs;        // kept substeps of the batch: [slot][kLegFields][32 pairs]
  float4* base;        // [slot][kBaseFields][8 pairs]
  float4* ckpt;        // states at the segment boundaries: slots as above, states only
  float* carry;        // [32][32 pairs] adjoint between segments
  float* part_cost;    // [N][G]
  float* part_grad;    // [N][G][13]
  unsigned long long* n_bad;

  __device__ __forceinline__ Kept kept(long long local, int lane) const {
    return Kept::of(legs, base, (size_t)pairs * 8, (size_t)local * 8 + (lane >> 2), lane & 3);
  }
  __device__ __forceinline__ Kept checkpoints(long long local, int lane) const {
    Kept k = kept(local, lane);
    k.leg = ckpt + local * 32 + lane;
    k.base = ckpt + (size_t)pairs * 32 * kLegFields * ((H - 1) / kSegSteps) + local * 8 + (lane >> 2);
    return k;
  }
};

// Where a warp's pair lies: its theta, windows and lanes.
struct PairLane {
  long long local;
  int n, g, lane, leg, w;
  bool active;
  __device__ __forceinline__ PairLane(const AdjArgs& a) {
    local = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const long long pair = a.pair0 + local;
    n = (int)(pair / a.G);
    g = (int)(pair % a.G);
    lane = threadIdx.x & 31;
    leg = lane & 3;
    w = g * 8 + (lane >> 2);
    active = w < a.win.W;
    if (!active) w = a.win.W - 1;
  }
};

// Control steps h0 .. h1 - 1. DETAIL: keep every substep (slot 0 is the first of h0) and the state at h1;
// otherwise only the states at the segment boundaries kSegSteps, 2 kSegSteps, .. < H.
// Bound by FP32 issue (75 % of the slots at 16 warps per SM); its stores ride along (0.12 cycles an issue).
template <bool DETAIL>
__global__ void __launch_bounds__(128) adjoint_forward_kernel(const DevModel* __restrict__ model, const AdjArgs a) {
  __shared__ DevModel M;
  load_model_smem(&M, model);
  __syncthreads();
  const PairLane P(a);
  if (P.local >= a.pairs) return;                   // uniform per warp
  const int W = a.win.W, dec = M.decimation, leg = P.leg, w = P.w;
  float th[SPI_THETA_DIM];
#pragma unroll
  for (int i = 0; i < SPI_THETA_DIM; ++i) th[i] = __ldg(a.theta + (size_t)P.n * SPI_THETA_DIM + i);
  const BaseParams<float> bp = base_params<float>(M, th);
  const LegParams<float> lp = leg_params<float>(th, leg);
  BaseState<float> B;
  LegState<float> L;
  if (DETAIL && a.h0 > 0) {
    adj::SolveWork<float> W0;
    Factor6 f0;
    SV<float> a00;
    load_kept<false>(a.checkpoints(P.local, P.lane), a.h0 / kSegSteps - 1, B, L, W0, f0, a00);
  } else {
    float s13[13];
#pragma unroll
    for (int i = 0; i < 13; ++i) s13[i] = __ldg(a.win.init + i * W + w);
    base_from_world(B, s13);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      L.q[k] = __ldg(a.win.init + (13 + 3 * leg + k) * W + w);
      L.qd[k] = __ldg(a.win.init + (25 + 3 * leg + k) * W + w);
    }
  }
  const Kept kept = a.kept(P.local, P.lane);
  const float none[3] = {0.f, 0.f, 0.f};
  for (int h = a.h0; h < a.h1; ++h) {
    if (!DETAIL && h > 0 && h % kSegSteps == 0) {
      const Kept c = a.checkpoints(P.local, P.lane);
      const int slot = h / kSegSteps - 1;
      keep_state(c, slot, leg, B);
      if (leg == 0) *c.base_at(slot, 3) = make_float4(B.nu.v.z, 0.f, 0.f, 0.f);
      keep_legs(c, slot, none, L);
    }
    float act[3];
    const float* ap = a.win.act + ((size_t)h * W + w) * 12 + 3 * leg;
    act[0] = __ldg(ap); act[1] = __ldg(ap + 1); act[2] = __ldg(ap + 2);
    for (int s = 0; s < dec; ++s) {
      if (DETAIL) substep_kept(M, leg, B, L, bp, lp, act, kept, (h - a.h0) * dec + s);
      else substep(M, leg, B, L, bp, lp, act);
    }
  }
  if (DETAIL) {
    const int slot = (a.h1 - a.h0) * dec;
    keep_state(kept, slot, leg, B);
    if (leg == 0) *kept.base_at(slot, 3) = make_float4(B.nu.v.z, 0.f, 0.f, 0.f);
    keep_legs(kept, slot, none, L);
  }
}

// Bound by its arithmetic at the 8 warps per SM that 255 registers leave (62 % of the issue slots). As one kernel
// with the forward pass, each substep computed again from its state, it waited for instructions 2.5
// cycles an issue: 13.4 ms for 512 theta x 256 windows x H = 20, 6.15 ms as two. The kept fields come
// straight from memory; staged a substep ahead in shared memory they took the same time.
__global__ void __launch_bounds__(128) adjoint_reverse_kernel(const DevModel* __restrict__ model, const AdjArgs a) {
  __shared__ DevModel M;
  load_model_smem(&M, model);
  __syncthreads();
  const PairLane P(a);
  if (P.local >= a.pairs) return;                   // uniform per warp
  const WinView& win = a.win;
  const int W = win.W, dec = M.decimation, leg = P.leg, lane = P.lane, w = P.w, n = P.n, g = P.g;
  const bool active = P.active;
  float th[SPI_THETA_DIM];
#pragma unroll
  for (int i = 0; i < SPI_THETA_DIM; ++i) th[i] = __ldg(a.theta + (size_t)n * SPI_THETA_DIM + i);
  const BaseParams<float> bp = base_params<float>(M, th);
  const LegParams<float> lp = leg_params<float>(th, leg);
  const Kept kept = a.kept(P.local, lane);
  adj::SolveWork<float> sw;
  Factor6 fac;
  SV<float> a0;
  BaseState<float> B;                               // the state after the substep at hand
  LegState<float> L;
  load_kept<false>(kept, (a.h1 - a.h0) * dec, B, L, sw, fac, a0);
  float* carry = a.carry + P.local * 32 + lane;
  const size_t cs = (size_t)a.pairs * 32;
  adj::BaseAdj<float> lam;
  float lq[3], lqd[3], gth[SPI_THETA_DIM], cost = 0.f;
  if (a.h1 == a.H) {
    // final cost and its adjoint
    float s13[13], tg13[13];
    base_to_world(B, s13);
#pragma unroll
    for (int i = 0; i < 13; ++i) tg13[i] = __ldg(win.tgt + i * W + w);
    float d13[13], sb13[13];
#pragma unroll
    for (int i = 0; i < 13; ++i) { d13[i] = s13[i] - tg13[i]; sb13[i] = 0.f; }
    float dq[3], dqd[3];
    bool finite = true;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      dq[k] = L.q[k] - __ldg(win.tgt + (13 + 3 * leg + k) * W + w);
      dqd[k] = L.qd[k] - __ldg(win.tgt + (25 + 3 * leg + k) * W + w);
      finite = finite && isfinite(L.q[k]) && isfinite(L.qd[k]);
      lq[k] = 0.f;
      lqd[k] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < 13; ++i) finite = finite && isfinite(s13[i]);
    if (a.mode == 1) {
      const float wq[6] = {a.w[0], a.w[1], a.w[2], a.w[3], a.w[4], a.w[5]};
      float base = 0.f;
#pragma unroll
      for (int i = 0; i < 13; ++i) {
        const float wi = i < 3 ? wq[0] : (i < 7 ? wq[1] : (i < 10 ? wq[2] : wq[3]));
        base += wi * d13[i] * d13[i];
        sb13[i] = 2.f * wi * d13[i];
      }
      float legs = 0.f;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        legs += wq[4] * dq[k] * dq[k] + wq[5] * dqd[k] * dqd[k];
        lq[k] = 2.f * wq[4] * dq[k];
        lqd[k] = 2.f * wq[5] * dqd[k];
      }
      cost = base + qsum(legs);
    } else {
      float np = 0.f, nq = 0.f, nj = 0.f;
#pragma unroll
      for (int i = 0; i < 3; ++i) np += d13[i] * d13[i];
#pragma unroll
      for (int i = 3; i < 7; ++i) nq += d13[i] * d13[i];
#pragma unroll
      for (int k = 0; k < 3; ++k) nj += dq[k] * dq[k];
      np = sqrtf(np); nq = sqrtf(nq); nj = sqrtf(qsum(nj));
      cost = 10.f * np + 5.f * nq + nj;
#pragma unroll
      for (int i = 0; i < 3; ++i) sb13[i] = np > 0.f ? 10.f * d13[i] / np : 0.f;
#pragma unroll
      for (int i = 3; i < 7; ++i) sb13[i] = nq > 0.f ? 5.f * d13[i] / nq : 0.f;
#pragma unroll
      for (int k = 0; k < 3; ++k) lq[k] = nj > 0.f ? dq[k] / nj : 0.f;
    }
    const float bad = qsum(finite ? 0.f : 1.f);
    if (active && leg == 0 && bad > 0.f) atomicAdd(a.n_bad, 1ull);
    lam = adj::base_to_world_bar(B, sb13);
#pragma unroll
    for (int i = 0; i < SPI_THETA_DIM; ++i) gth[i] = 0.f;
  } else {
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = carry[i * cs];
    lam.p = v3(v[0], v[1], v[2]);
    lam.qx = v[3]; lam.qy = v[4]; lam.qz = v[5]; lam.qw = v[6];
    lam.nu.w = v3(v[7], v[8], v[9]);
    lam.nu.v = v3(v[10], v[11], v[12]);
#pragma unroll
    for (int k = 0; k < 3; ++k) { lq[k] = v[13 + k]; lqd[k] = v[16 + k]; }
#pragma unroll
    for (int i = 0; i < SPI_THETA_DIM; ++i) gth[i] = v[19 + i];
  }
  for (int h = a.h1 - 1; h >= a.h0; --h) {
    float act[3];
    const float* ap = win.act + ((size_t)h * W + w) * 12 + 3 * leg;
    act[0] = __ldg(ap); act[1] = __ldg(ap + 1); act[2] = __ldg(ap + 2);
    for (int s = dec - 1; s >= 0; --s) {
      BaseState<float> B0;
      LegState<float> L0;
      load_kept<true>(kept, (h - a.h0) * dec + s, B0, L0, sw, fac, a0);
      substep_adjoint(M, leg, B0, L0, B, sw, fac, a0, bp, lp, th, act, lam, lq, lqd, gth);
      B = B0;
    }
  }
  if (a.h1 == a.H) {
    const float wt = active ? __ldg(win.weight + w) : 0.f;
    cost = slot_sum(leg == 0 ? cost * wt : 0.f);
    if (lane == 0) a.part_cost[(size_t)n * a.G + g] = cost;
  }
  if (a.h0 > 0) {
    const float v[19] = {lam.p.x, lam.p.y, lam.p.z, lam.qx, lam.qy, lam.qz, lam.qw, lam.nu.w.x, lam.nu.w.y, lam.nu.w.z,
                         lam.nu.v.x, lam.nu.v.y, lam.nu.v.z, lq[0], lq[1], lq[2], lqd[0], lqd[1], lqd[2]};
#pragma unroll
    for (int i = 0; i < 19; ++i) carry[i * cs] = v[i];
#pragma unroll
    for (int i = 0; i < SPI_THETA_DIM; ++i) carry[(19 + i) * cs] = gth[i];
    return;
  }
  // window-weighted sums over the warp's 8 windows
  const float wt = active ? __ldg(win.weight + w) : 0.f;
#pragma unroll
  for (int i = 0; i < SPI_THETA_DIM; ++i) gth[i] = slot_sum(qsum(gth[i]) * wt);
  if (lane == 0) {
#pragma unroll
    for (int i = 0; i < SPI_THETA_DIM; ++i) a.part_grad[((size_t)n * a.G + g) * SPI_THETA_DIM + i] = gth[i];
  }
}

__global__ void adjoint_finalize(const float* __restrict__ part_cost, const float* __restrict__ part_grad, int N,
                                 int G, float norm, float* __restrict__ cost, float* __restrict__ grad) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  float c = 0.f, gr[SPI_THETA_DIM];
#pragma unroll
  for (int i = 0; i < SPI_THETA_DIM; ++i) gr[i] = 0.f;
  for (int g = 0; g < G; ++g) {
    c += part_cost[(size_t)n * G + g];
#pragma unroll
    for (int i = 0; i < SPI_THETA_DIM; ++i) gr[i] += part_grad[((size_t)n * G + g) * SPI_THETA_DIM + i];
  }
  const float inv = 1.0f / norm;
  if (cost) cost[n] = c * inv;
  if (grad) {
#pragma unroll
    for (int i = 0; i < SPI_THETA_DIM; ++i) grad[(size_t)n * SPI_THETA_DIM + i] = gr[i] * inv;
  }
}

}  // namespace

extern "C" int spi_adjoint(spi_engine* e, const float* theta, int N, float* cost, float* grad) {
  if (!e || !theta) return set_error(SPI_EINVAL, "spi_adjoint: null argument");
  if (N <= 0) return set_error(SPI_EINVAL, "spi_adjoint: N=%d must be > 0", N);
  if (e->W <= 0 || e->H <= 0) return set_error(SPI_ESTATE, "spi_adjoint before spi_load_windows");
  const int G = (e->W + 7) / 8, dec = e->host_model.decimation, H = e->H;
  const long long all = (long long)N * G;
  const int seg = std::min(H, kSegSteps), bounds = (H - 1) / kSegSteps;   // boundaries inside the horizon
  const size_t slots = (size_t)seg * dec + 1;
  // batches of equal size within the engine's limit; smaller ones when the device has less to give
  long long batch;
  int rc;
  for (e->adj_limit.begin_call();; e->adj_limit.refused(slots * batch * kPairBytes)) {
    const long long most = std::max(1LL, (long long)(e->adj_limit.bytes / (slots * kPairBytes)));
    const long long batches = (all + most - 1) / most;
    batch = (all + batches - 1) / batches;
    rc = e->adj_seg.reserve(slots * batch * kPairBytes);
    if (!rc) rc = e->adj_ckpt.reserve(bounds * batch * (kPairBytes + (size_t)32 * 32 * sizeof(float)));
    if (rc != SPI_ENOMEM || batch == 1) break;
  }
  if (rc == SPI_ENOMEM) e->adj_limit = ScratchLimit();   // nothing to be had: the next call begins anew
  if (!rc) rc = e->adj_part.reserve((size_t)all * (SPI_THETA_DIM + 1) * sizeof(float));
  if (rc) return rc;
  AdjArgs a;
  a.win = WinView{e->init.f(), e->act.f(), e->tgt.f(), e->weight.f(), e->W, e->H};
  a.theta = theta;
  a.G = G;
  a.mode = e->cost_mode;
  for (int i = 0; i < 6; ++i) a.w[i] = e->sq_w[i];
  a.H = H;
  a.part_cost = e->adj_part.f();
  a.part_grad = e->adj_part.f() + (size_t)all;
  a.n_bad = (unsigned long long*)e->bad.p;
  for (long long p0 = 0; p0 < all; p0 += batch) {
    a.pair0 = p0;
    a.pairs = std::min(batch, all - p0);
    a.legs = (float4*)e->adj_seg.p;
    a.base = a.legs + slots * kLegFields * 32 * a.pairs;
    a.ckpt = (float4*)e->adj_ckpt.p;
    a.carry = (float*)(a.ckpt + (size_t)bounds * (kLegFields * 32 + kBaseFields * 8) * a.pairs);
    const unsigned grid = blocks_for(a.pairs, 4);
    if (bounds > 0) {
      a.h0 = 0;
      a.h1 = bounds * kSegSteps + 1;     // the last boundary's state is kept before its step runs
      adjoint_forward_kernel<false><<<grid, 128, 0, e->stream>>>(e->d_model, a);
    }
    for (int c = bounds; c >= 0; --c) {
      a.h0 = c * kSegSteps;
      a.h1 = std::min(H, a.h0 + kSegSteps);
      adjoint_forward_kernel<true><<<grid, 128, 0, e->stream>>>(e->d_model, a);
      adjoint_reverse_kernel<<<grid, 128, 0, e->stream>>>(e->d_model, a);
    }
    const cudaError_t le = cudaGetLastError();
    if (le != cudaSuccess) return cuda_error(le, "spi_adjoint: rollout launch");
  }
  adjoint_finalize<<<blocks_for(N, 128), 128, 0, e->stream>>>(a.part_cost, a.part_grad, N, G, e->norm, cost, grad);
  const cudaError_t ce = cudaGetLastError();
  if (ce != cudaSuccess) return cuda_error(ce, "spi_adjoint: finalize launch");
  return SPI_OK;
}
