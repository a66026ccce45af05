// eval.cu -- rollouts of a caller's theta batch (spi_run after spi_set_theta).
//
// Work is a flat list of (theta n, eight-window group g) pairs, n G + g. Two kernels with the
// same bits (rollout_hip.cuh):
//   eval_lane_kernel  a warp takes four pairs, one lane per window;
//   eval_team_kernel  a warp takes one pair, four lanes per window.
// The engine CEM and the server keep the kernels of items.cu: a search's path turns on which of
// two near-equal costs ranks first, so their costs stay bit for bit what they were.
#include <cuda_runtime.h>

#include "eval.h"
#include "rollout_hip.cuh"

namespace spi {
namespace {

// Issue-bound: 2,900 warp instructions a substep (84 % FP32) at 12 warps per SM, 78 % of the issue slots
// used, the FP32 pipe 66 % busy. 4096 theta x 256 windows x H = 20: 7.87 ms; 8.92 ms with phase A of
// dynamics.cuh (3,710 instructions).
template <int MINB, int MS>
__global__ void __launch_bounds__(128, MINB) eval_lane_kernel(const __grid_constant__ EvalModel M, const EvalArgs a) {
  extern __shared__ float4 lane_smem[];              // kHipSlotBytes
  __shared__ BaseParams<float> bp_warp[4][4];
  __shared__ float4 gains_warp[4][4][8];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, grp = lane >> 3, sub = lane & 7;
  const long long pairs = (long long)a.N * a.G;
  long long q = ((long long)blockIdx.x * 4 + wib) * 4;
  if (q >= pairs) return;                            // uniform per warp; no CTA barrier below
  q += grp;
  const bool live = q < pairs;
  if (!live) q = pairs - 1;
  const int W = a.win.W, H = a.win.H;
  const int n = (int)(q / a.G), g = (int)(q % a.G);
  const int w = min(g * 8 + sub, W - 1);             // this lane's window (clamped into the set)
  const bool active = live && g * 8 + sub < W;
  {
    float th[SPI_THETA_DIM];
#pragma unroll
    for (int i = 0; i < SPI_THETA_DIM; ++i) th[i] = __ldg(a.theta + (size_t)n * SPI_THETA_DIM + i);
    if (sub == 0) bp_warp[wib][grp] = base_params<float>(M, th);
    if (sub < 4) store_gains(leg_gains(M, leg_params<float>(th, sub), sub), gains_warp[wib][grp] + 2 * sub);
    __syncwarp();
  }
  const HipSlots sl{lane_smem + threadIdx.x};
  const float no_error[2] = {0.f, 0.f};
  V3<float> pe = v3(0.f, 0.f, 0.f);
  BaseState<float> B;
  {
    float s13[13];
#pragma unroll
    for (int i = 0; i < 13; ++i) s13[i] = __ldg(a.win.init + i * W + w);
    base_from_world(B, s13);
    pin(B);
#pragma unroll
    for (int leg = 0; leg < 4; ++leg) {
      LegState<float> L;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        L.q[k] = __ldg(a.win.init + (13 + 3 * leg + k) * W + w);
        L.qd[k] = __ldg(a.win.init + (25 + 3 * leg + k) * W + w);
      }
      sl.put_leg_state(leg, L, no_error);
    }
  }
  for (int h = 0; h < H; ++h) {
    const float4* ap = reinterpret_cast<const float4*>(a.win.act + ((size_t)h * W + w) * 12);
    sl.put_targets(M, __ldg(ap), __ldg(ap + 1), __ldg(ap + 2));
    for (int s = 0; s < M.decimation; ++s) substep_hip_lane<MS>(M, B, pe, sl, &bp_warp[wib][grp], gains_warp[wib][grp]);
  }
  LegState<float> L[4];
#pragma unroll
  for (int leg = 0; leg < 4; ++leg) {
    float e[2];
    L[leg] = sl.leg_state(leg, e);
  }
  float s13[13];
  base_to_world(B, s13);
  window_result(a.win, w, active, s13, L, live ? a.partial + (size_t)q * SPI_N_COMP : nullptr, a.n_bad);
}

// Latency-bound: one chain of substeps per rollout, at most a few warps per scheduler (0.43 of the issue slots of an SM
// with one CTA). 64 theta x 8 windows x H = 5: 26 us for the launch and its finalize, against 57 us with
// one lane per rollout.
template <int MS>
__global__ void __launch_bounds__(128) eval_team_kernel(const __grid_constant__ EvalModel M, const EvalArgs a) {
  __shared__ TeamShare share_cta[4];
  __shared__ HipLeg<float> hip[4];
  stage_hip(hip, M);
  const long long q = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (q >= (long long)a.N * a.G) return;             // uniform per warp; no CTA barrier below
  const int n = (int)(q / a.G), g = (int)(q % a.G);
  const int lane = threadIdx.x & 31, leg = lane & 3;
  const int W = a.win.W, H = a.win.H;
  const int w = min(g * 8 + (lane >> 2), W - 1);     // this team's window (clamped into the set)
  TeamShare& share = share_cta[threadIdx.x >> 5];
  TeamRollout R;
  R.init(M, share, a.win.init + w, W, a.theta + (size_t)n * SPI_THETA_DIM);
  const float* ap = a.win.act + (size_t)w * 12 + 3 * leg;
  for (int h = 0; h < H; ++h) {
    float tgt[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) tgt[k] = joint_target(M, k, leg, __ldg(ap + (size_t)h * W * 12 + k));
    for (int s = 0; s < M.decimation; ++s) R.substep<MS>(M, hip + leg, tgt, share);
  }
  // the final state to one lane per window (lanes 0..7 of the warp; the others compute copies)
  float s13[13];
  base_to_world(R.B, s13);
  const int src = (lane & 7) * 4;
#pragma unroll
  for (int i = 0; i < 13; ++i) s13[i] = __shfl_sync(0xffffffffu, s13[i], src);
  LegState<float> L[4];
#pragma unroll
  for (int l = 0; l < 4; ++l)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      L[l].q[k] = __shfl_sync(0xffffffffu, R.L.q[k], src + l);
      L[l].qd[k] = __shfl_sync(0xffffffffu, R.L.qd[k], src + l);
    }
  const int wf = g * 8 + (lane & 7);
  window_result(a.win, min(wf, W - 1), lane < 8 && wf < W, s13, L,
                lane < 8 ? a.partial + (size_t)q * SPI_N_COMP : nullptr, a.n_bad);
}

// Whether a launch of `pairs` (theta, group) pairs is faster in the team form. A CTA carries 4 pairs as
// teams and 16 in the lane form, and a launch takes as long as its fullest SM. Measured at H = 20
// (80 substeps), microseconds by CTAs on the fullest SM: team 81, 115, 154, 247, 251, 294 (1..6; three are
// resident), lane 204, 334, 447 (1..3). So up to three team CTAs beat one lane CTA, and five or six (a
// launch that would need two lane CTAs) beat two.
bool use_team(long long pairs, int sms) {
  const long long team = (pairs + 4LL * sms - 1) / (4LL * sms), lane = (pairs + 16LL * sms - 1) / (16LL * sms);
  return team <= 3 || (lane == 2 && team <= 6);
}

// The register cap that min_blocks asks for, up to three CTAs per SM: more do not fit beside their 72 KB of shared
// memory, and the cap of four (128 registers) costs the 148-register kernel 48 bytes of spills for nothing
// (2048 theta x 64 windows x H = 20: 1,059 us at three, 1,092 under that cap).
const void* lane_kernel(int min_blocks, bool sl) {
  if (min_blocks <= 2)
    return sl ? (const void*)eval_lane_kernel<2, kMotorSpeedLimit> : (const void*)eval_lane_kernel<2, kMotorRuntime>;
  return sl ? (const void*)eval_lane_kernel<3, kMotorSpeedLimit> : (const void*)eval_lane_kernel<3, kMotorRuntime>;
}

}  // namespace

cudaError_t eval_prepare() {
  for (int mb = 2; mb <= 3; ++mb)
    for (bool sl : {false, true}) {
      const cudaError_t ce =
          cudaFuncSetAttribute(lane_kernel(mb, sl), cudaFuncAttributeMaxDynamicSharedMemorySize, kHipSlotBytes);
      if (ce != cudaSuccess) return ce;
    }
  return cudaSuccess;
}

cudaError_t eval_launch(const EvalModel& model, int min_blocks, int sms, const EvalArgs& a, cudaStream_t stream) {
  const bool sl = motor_shape_of(model) == kMotorSpeedLimit;
  const long long pairs = (long long)a.N * a.G;
  const void* func;
  long long grid;
  unsigned smem = 0;
  if (use_team(pairs, sms)) {
    grid = (pairs + 3) / 4;
    func = sl ? (const void*)eval_team_kernel<kMotorSpeedLimit> : (const void*)eval_team_kernel<kMotorRuntime>;
  } else {
    grid = (pairs + 15) / 16;
    func = lane_kernel(min_blocks, sl);
    smem = kHipSlotBytes;
  }
  if (grid > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  void* args[] = {(void*)&model, (void*)&a};
  return cudaLaunchKernel(func, dim3((unsigned)grid), dim3(128), args, smem, stream);
}

}  // namespace spi
