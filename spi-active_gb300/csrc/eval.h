// eval.h -- the rollout kernels of spi_run on a caller's theta batch (eval.cu).
#pragma once

#include <cuda_runtime.h>

#include "leg_hip.cuh"
#include "rollout.cuh"

namespace spi {

struct EvalArgs {
  WinView win;
  const float* theta;          // [N][SPI_THETA_DIM]
  float* partial;              // [N][G][SPI_N_COMP]
  int N, G;                    // theta samples; eight-window groups, ceil(W / 8)
  unsigned long long* n_bad;
};

// Raise the dynamic shared-memory limit of the lane-form kernels.
cudaError_t eval_prepare();
// Launch the rollouts of `a` on a GPU of `sms` SMs. min_blocks: the lane form's register cap (2: 255
// registers, 3 and more: 168).
cudaError_t eval_launch(const EvalModel& model, int min_blocks, int sms, const EvalArgs& a, cudaStream_t stream);

}  // namespace spi
