// windows.cuh -- windows from the caller's row layout to the kernels' structure of arrays.
#pragma once

#include <cuda_runtime.h>

#include "spi_engine.h"

namespace spi {

// init and target [W][37] -> [37][W], actions [W][H][12] -> [H][W][12], weight [W] (null: all 1), in one
// launch: a window set is a few hundred KB, so the call is its launches (18 us against 23 with one for each array).
// The first state_blocks CTAs take the states and weights, the others the actions, one value a thread; with both
// in one loop 70,000 windows x 20 steps took 127 us, 99 as four launches.
static __global__ void pack_windows_kernel(const float* __restrict__ init, const float* __restrict__ actions,
                                           const float* __restrict__ target, const float* __restrict__ weight, int W, int H,
                                           unsigned state_blocks, float* __restrict__ d_init, float* __restrict__ d_act,
                                           float* __restrict__ d_tgt, float* __restrict__ d_weight) {
  if (blockIdx.x < state_blocks) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < (long long)W * SPI_STATE_DIM) {
      const size_t at = (size_t)(i % SPI_STATE_DIM) * W + (size_t)(i / SPI_STATE_DIM);
      d_init[at] = init[i];
      d_tgt[at] = target[i];
    }
    if (i < W) d_weight[i] = weight ? weight[i] : 1.0f;
  } else {
    const long long i = (long long)(blockIdx.x - state_blocks) * blockDim.x + threadIdx.x;
    if (i >= (long long)W * H * 12) return;
    const int j = (int)(i % 12);
    const long long wh = i / 12;
    const int h = (int)(wh % H), w = (int)(wh / H);
    d_act[((size_t)h * W + w) * 12 + j] = actions[i];
  }
}

inline cudaError_t pack_windows(const float* init, const float* actions, const float* target, const float* weight, int W,
                                int H, float* d_init, float* d_act, float* d_tgt, float* d_weight, cudaStream_t stream) {
  const unsigned states = (unsigned)(((long long)W * SPI_STATE_DIM + 255) / 256);
  const unsigned acts = (unsigned)(((long long)W * H * 12 + 255) / 256);
  pack_windows_kernel<<<states + acts, 256, 0, stream>>>(init, actions, target, weight, W, H, states, d_init, d_act, d_tgt,
                                                        d_weight);
  return cudaGetLastError();
}

}  // namespace spi
