// windows.cuh -- windows from the caller's row layout to the kernels' structure of arrays.
#pragma once

#include <cuda_runtime.h>

#include "spi_engine.h"

namespace spi {

// init and target [W][37] -> [37][W], actions [W][H][12] -> [H][W][12], weight [W] (null: all 1), in one
// launch: a window set is a few hundred KB, so the call is its launches.
static __global__ void pack_windows_kernel(const float* __restrict__ init, const float* __restrict__ actions,
                                           const float* __restrict__ target, const float* __restrict__ weight, int W, int H,
                                           float* __restrict__ d_init, float* __restrict__ d_act,
                                           float* __restrict__ d_tgt, float* __restrict__ d_weight) {
  const long long ns = (long long)W * SPI_STATE_DIM, na = (long long)W * H * 12;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < na; i += (long long)gridDim.x * blockDim.x) {
    const int j = (int)(i % 12);
    const long long wh = i / 12;
    const int h = (int)(wh % H), w = (int)(wh / H);
    d_act[((size_t)h * W + w) * 12 + j] = actions[i];
    if (i < ns) {
      const int f = (int)(i % SPI_STATE_DIM);
      const size_t at = (size_t)f * W + (size_t)(i / SPI_STATE_DIM);
      d_init[at] = init[i];
      d_tgt[at] = target[i];
    }
    if (i < W) d_weight[i] = weight ? weight[i] : 1.0f;
  }
  // (a horizon under four control steps has fewer action values than a state row)
  for (long long i = na + (long long)blockIdx.x * blockDim.x + threadIdx.x; i < ns; i += (long long)gridDim.x * blockDim.x) {
    const int f = (int)(i % SPI_STATE_DIM);
    const size_t at = (size_t)f * W + (size_t)(i / SPI_STATE_DIM);
    d_init[at] = init[i];
    d_tgt[at] = target[i];
  }
}

inline cudaError_t pack_windows(const float* init, const float* actions, const float* target, const float* weight, int W,
                                int H, float* d_init, float* d_act, float* d_tgt, float* d_weight, cudaStream_t stream) {
  const long long n = (long long)W * (H * 12LL > SPI_STATE_DIM ? H * 12LL : SPI_STATE_DIM);
  const long long grid = (n + 255) / 256;
  pack_windows_kernel<<<(unsigned)(grid < 65536 ? grid : 65536), 256, 0, stream>>>(init, actions, target, weight, W, H,
                                                                                  d_init, d_act, d_tgt, d_weight);
  return cudaGetLastError();
}

}  // namespace spi
