// engine_impl.h -- the engine object behind the opaque spi_engine handle.
#pragma once

#include <cuda_runtime.h>

#include "cem_state.h"
#include "common.h"
#include "leg_hip.cuh"

struct spi_engine {
  spi::EvalModel host_model;
  spi::DevModel* d_model = nullptr;
  int sms = 0;                             // SMs of the engine's device
  cudaStream_t stream = nullptr;
  spi::DeviceBuf init, act, tgt, weight;   // windows, structure-of-arrays
  int W = 0, H = 0;
  float norm = 1.f;
  spi::DeviceBuf theta;                    // [N][13]
  int N = 0;
  bool population = false;                 // the batch is the CEM's population (spi_run keeps its kernels)
  spi::DeviceBuf partial, comp, cost;      // [N][G][9], [N][9], [N]
  spi::DeviceBuf bad;                      // one unsigned long long
  int cost_mode = 1;
  float sq_w[6] = {10.f, 5.f, 0.1f, 0.1f, 1.f, 0.01f};
  bool ran = false;
  // rollout kernel of a caller's theta batch and of the CEM's population: lane layout, occupancy variant
  struct { int layout = 0, min_blocks = 3; } kernel[2];
  spi::DeviceBuf items;                    // one-slot work table of the rollout kernel (items.h)
  // CEM
  spi::DeviceBuf cem;                      // one CemState
  bool cem_ready = false;
  int cem_n = 0;                           // CEM population size
  cudaGraphExec_t graph_exec = nullptr;
  cudaStream_t capture_stream = nullptr;   // graphs are captured here, replayed on `stream`
  unsigned seen_generation = 0;            // buffer generations the graph / CEM pointers refer to
  spi::DeviceBuf sens_kept;                // kept substeps of the sensitivities' first direction
  spi::ScratchLimit sens_limit;
  cudaEvent_t sens_done = nullptr;         // after the last call that used sens_kept
  spi::DeviceBuf adj_ckpt, adj_seg, adj_part;   // adjoint checkpoints, kept substeps, partials
  spi::ScratchLimit adj_limit;             // of adj_seg
};

namespace spi {
// population: with the kernels of the CEM's population (trace: neither's)
int run_impl(spi_engine* e, float* trace, bool population);
// The buffers of a run over the engine's theta batch; what depends on their addresses follows them.
int reserve_run(spi_engine* e);
// Call after any DeviceBuf::reserve of theta / cost / partial / comp / windows: if one of
// them moved, drops the captured CEM graph and points the device CEM state at the new
// theta / cost buffers.
int refresh_after_realloc(spi_engine* e);
// Raise the tangent kernels' dynamic shared-memory limit to what any number of directions needs. The limit belongs to
// the kernel, not to an engine or a call: it is set to the same value by every engine, never per call.
cudaError_t sensitivity_prepare();
inline unsigned blocks_for(long long n, int t) { return (unsigned)((n + t - 1) / t); }
}  // namespace spi
