// engine.cu -- C ABI of the batched candidate-evaluation engine (declared in spi_engine.h).
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <string>

#include "common.h"
#include "engine_impl.h"
#include "eval.h"
#include "items.h"
#include "model.h"
#include "rollout.cuh"
#include "rollout_block.cuh"
#include "windows.cuh"

using namespace spi;

namespace spi {
thread_local std::string g_last_error;
int set_error(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  g_last_error = buf;
  return code;
}
int cuda_error(cudaError_t e, const char* what) {
  return set_error(SPI_ECUDA, "%s: %s", what, cudaGetErrorString(e));
}
}  // namespace spi

namespace {

// finalize_costs for spi_evaluate, in the same launch to the caller's outputs and with the theta batch
// kept as the engine's own: the call has no copies to wait for.
__global__ void finalize_evaluate(const float* __restrict__ partial, int N, int G, float norm, int mode, float w0,
                                  float w1, float w2, float w3, float w4, float w5, const float* __restrict__ theta,
                                  float* __restrict__ own_theta, float* __restrict__ own_comp,
                                  float* __restrict__ own_cost, float* __restrict__ comp, float* __restrict__ cost) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  const float w[6] = {w0, w1, w2, w3, w4, w5};
  finalize_one(partial, n, G, norm, mode, w, own_comp, own_cost);
#pragma unroll
  for (int i = 0; i < SPI_THETA_DIM; ++i) own_theta[(size_t)n * SPI_THETA_DIM + i] = theta[(size_t)n * SPI_THETA_DIM + i];
  if (comp) {
#pragma unroll
    for (int k = 0; k < SPI_N_COMP; ++k) comp[(size_t)n * SPI_N_COMP + k] = own_comp[(size_t)n * SPI_N_COMP + k];
  }
  if (cost) cost[n] = own_cost[n];
}

// Room for N theta samples. Without it the batch that the engine had is gone too.
int reserve_theta(spi_engine* e, int N) {
  const int rc = e->theta.reserve((size_t)N * SPI_THETA_DIM * 4);
  if (rc) { e->N = 0; e->ran = false; }
  return rc;
}

int check_kernel(const char* what, int layout, int min_blocks) {
  if (layout != SPI_LAYOUT_QUAD && layout != SPI_LAYOUT_LANE && layout != SPI_LAYOUT_BLOCK)
    return set_error(SPI_EINVAL, "%s: layout %d not 0/1/2", what, layout);
  const int lo = layout == SPI_LAYOUT_LANE ? 2 : 3;
  if (min_blocks < lo || min_blocks > 5)
    return set_error(SPI_EINVAL, "%s: min_blocks %d outside [%d, 5]", what, min_blocks, lo);
  return SPI_OK;
}
int prepare_kernel(const char* what, int layout) {
  if (layout != SPI_LAYOUT_LANE) return SPI_OK;
  // the parking area is above the 48 KB default for dynamic shared memory
  cudaError_t ce = items_prepare_lane();
  if (ce == cudaSuccess) ce = eval_prepare();
  return ce == cudaSuccess ? SPI_OK : cuda_error(ce, what);
}

}  // namespace

int spi::reserve_run(spi_engine* e) {
  const int G = (e->W + 7) / 8;
  int rc = e->partial.reserve((size_t)e->N * G * SPI_N_COMP * sizeof(float));
  if (!rc) rc = e->comp.reserve((size_t)e->N * SPI_N_COMP * sizeof(float));
  if (!rc) rc = e->cost.reserve((size_t)e->N * sizeof(float));
  if (rc) e->ran = false;   // a buffer that could not grow is gone
  return rc ? rc : refresh_after_realloc(e);
}

int spi::run_impl(spi_engine* e, float* trace, bool population) {
  if (!e) return set_error(SPI_EINVAL, "null engine");
  if (e->W <= 0 || e->H <= 0) return set_error(SPI_ESTATE, "spi_run before spi_load_windows");
  if (e->N <= 0) return set_error(SPI_ESTATE, "spi_run before spi_set_theta");
  const int G = (e->W + 7) / 8;
  int rc = reserve_run(e);
  if (rc) return rc;
  WinView win{e->init.f(), e->act.f(), e->tgt.f(), e->weight.f(), e->W, e->H};
  const long long warps = (long long)e->N * G;
  const unsigned grid = blocks_for(warps, 4);
  unsigned long long* bad = (unsigned long long*)e->bad.p;
  const int layout = e->kernel[population].layout, min_blocks = e->kernel[population].min_blocks;
  if (trace) {
    rollout_kernel<true, 3><<<grid, 128, 0, e->stream>>>(e->d_model, win, e->theta.f(), e->N, G,
                                                         e->partial.f(), trace, bad);
  } else if (layout == SPI_LAYOUT_LANE && !population) {
    const EvalArgs a{win, e->theta.f(), e->partial.f(), e->N, G, bad};
    const cudaError_t ce = eval_launch(e->host_model, min_blocks, e->sms, a, e->stream);
    if (ce != cudaSuccess) return cuda_error(ce, "rollout launch");
  } else if (layout != SPI_LAYOUT_BLOCK) {
    // the server's rollout kernel on a table of one slot (items.h), one warp per work item
    SlotDesc d{};
    d.win = win;
    d.theta = e->theta.f();
    d.partial = e->partial.f();
    d.comp = e->comp.f();
    d.cost = e->cost.f();
    d.N = e->N;
    d.G = G;
    d.norm = e->norm;
    d.active = 1;
    const long long items = items_of(layout, e->N, G);
    const long long ctas = items_grid(items, 1);
    if (ctas > 0x7fffffffLL) return set_error(SPI_EINVAL, "spi_run: %lld work items", items);
    SingleTable* tab = static_cast<SingleTable*>(e->items.p);
    cudaError_t ce = items_fill_single(tab, d, items, 1, e->stream);
    if (ce == cudaSuccess)
      ce = items_launch(layout, min_blocks, e->host_model, e->d_model, single_tables(tab), 0, (int)ctas, bad,
                        e->stream);
    if (ce != cudaSuccess) return cuda_error(ce, "rollout launch");
  } else {
    if (min_blocks == 4)
      rollout_block_kernel<4><<<grid, 128, 0, e->stream>>>(e->d_model, win, e->theta.f(), e->N, G,
                                                            e->partial.f(), bad);
    else if (min_blocks == 5)
      rollout_block_kernel<5><<<grid, 128, 0, e->stream>>>(e->d_model, win, e->theta.f(), e->N, G,
                                                            e->partial.f(), bad);
    else
      rollout_block_kernel<3><<<grid, 128, 0, e->stream>>>(e->d_model, win, e->theta.f(), e->N, G,
                                                            e->partial.f(), bad);
  }
  cudaError_t ce = cudaGetLastError();
  if (ce != cudaSuccess) return cuda_error(ce, "rollout_kernel launch");
  const float* w = e->sq_w;
  finalize_costs<<<blocks_for(e->N, 128), 128, 0, e->stream>>>(e->partial.f(), e->N, G, e->norm,
                                                               e->cost_mode, w[0], w[1], w[2], w[3],
                                                               w[4], w[5], e->comp.f(), e->cost.f());
  ce = cudaGetLastError();
  if (ce != cudaSuccess) return cuda_error(ce, "finalize_costs launch");
  e->ran = true;
  return SPI_OK;
}

extern "C" {

int spi_abi_version(void) { return SPI_ABI_VERSION; }

const char* spi_last_error(void) { return g_last_error.c_str(); }

int spi_create(const spi_robot* robot, spi_engine** out) {
  if (!robot || !out) return set_error(SPI_EINVAL, "spi_create: null argument");
  *out = nullptr;
  spi_engine* e = new (std::nothrow) spi_engine();
  if (!e) return set_error(SPI_ENOMEM, "spi_create: host allocation failed");
  const char* why = "";
  int rc = build_eval_model(*robot, &e->host_model, &why);
  if (rc) { delete e; return set_error(rc, "spi_create: %s", why); }
  cudaError_t ce = cudaMalloc(&e->d_model, sizeof(DevModel));
  if (ce != cudaSuccess) { delete e; return cuda_error(ce, "spi_create: cudaMalloc(model)"); }
  ce = cudaMemcpy(e->d_model, static_cast<const DevModel*>(&e->host_model), sizeof(DevModel), cudaMemcpyHostToDevice);
  if (ce != cudaSuccess) { cudaFree(e->d_model); delete e; return cuda_error(ce, "spi_create: upload model"); }
  rc = e->bad.reserve(sizeof(unsigned long long));
  if (!rc) rc = e->items.reserve(sizeof(SingleTable));
  if (rc) { cudaFree(e->d_model); delete e; return rc; }
  cudaMemset(e->bad.p, 0, sizeof(unsigned long long));
  int dev = 0;
  ce = cudaGetDevice(&dev);
  if (ce == cudaSuccess) ce = cudaDeviceGetAttribute(&e->sms, cudaDevAttrMultiProcessorCount, dev);
  if (ce == cudaSuccess) ce = sensitivity_prepare();
  if (ce != cudaSuccess) { spi_destroy(e); return cuda_error(ce, "spi_create: device"); }
  // default kernel: the lane layout at the 168-register cap (the fastest on the C1 workload)
  if ((rc = spi_set_kernel_layout(e, SPI_LAYOUT_LANE)) || (rc = spi_set_kernel_config(e, 3))) {
    spi_destroy(e);
    return rc;
  }
  *out = e;
  return SPI_OK;
}

int spi_destroy(spi_engine* e) {
  if (!e) return SPI_OK;
  if (e->graph_exec) cudaGraphExecDestroy(e->graph_exec);
  if (e->capture_stream) cudaStreamDestroy(e->capture_stream);
  if (e->sens_done) cudaEventDestroy(e->sens_done);
  if (e->d_model) cudaFree(e->d_model);
  delete e;
  return SPI_OK;
}

int spi_set_stream(spi_engine* e, void* stream) {
  if (!e) return set_error(SPI_EINVAL, "null engine");
  e->stream = (cudaStream_t)stream;
  return SPI_OK;
}

int spi_load_windows(spi_engine* e, const float* init, const float* actions, const float* target,
                     const float* weight, int W, int H, float norm) {
  if (!e || !init || !actions || !target) return set_error(SPI_EINVAL, "spi_load_windows: null argument");
  if (W <= 0 || H <= 0) return set_error(SPI_EINVAL, "spi_load_windows: W=%d H=%d must be > 0", W, H);
  if ((long long)W * H * 12 > (1ll << 31)) return set_error(SPI_EINVAL, "spi_load_windows: too many window steps");
  int rc;
  if ((rc = e->init.reserve((size_t)W * SPI_STATE_DIM * 4))) return rc;
  if ((rc = e->tgt.reserve((size_t)W * SPI_STATE_DIM * 4))) return rc;
  if ((rc = e->act.reserve((size_t)W * H * 12 * 4))) return rc;
  if ((rc = e->weight.reserve((size_t)W * 4))) return rc;
  if ((rc = refresh_after_realloc(e))) return rc;
  const cudaError_t ce = pack_windows(init, actions, target, weight, W, H, e->init.f(), e->act.f(), e->tgt.f(),
                                      e->weight.f(), e->stream);
  if (ce != cudaSuccess) return cuda_error(ce, "spi_load_windows");
  e->W = W;
  e->H = H;
  e->norm = norm > 0.f ? norm : (float)W;
  e->ran = false;
  // a captured CEM iteration bakes in W, H and norm: capture again on next use
  if (e->graph_exec) { cudaGraphExecDestroy(e->graph_exec); e->graph_exec = nullptr; }
  return SPI_OK;
}

int spi_set_theta(spi_engine* e, const float* theta, int N) {
  if (!e || !theta) return set_error(SPI_EINVAL, "spi_set_theta: null argument");
  if (N <= 0) return set_error(SPI_EINVAL, "spi_set_theta: N=%d must be > 0", N);
  int rc = reserve_theta(e, N);
  if (rc) return rc;
  if ((rc = refresh_after_realloc(e))) return rc;
  cudaError_t ce = cudaMemcpyAsync(e->theta.p, theta, (size_t)N * SPI_THETA_DIM * 4,
                                   cudaMemcpyDeviceToDevice, e->stream);
  if (ce != cudaSuccess) return cuda_error(ce, "spi_set_theta");
  e->N = N;
  e->population = false;
  e->ran = false;
  return SPI_OK;
}

int spi_set_kernel_config(spi_engine* e, int min_blocks) {
  if (!e) return set_error(SPI_EINVAL, "null engine");
  for (const auto& k : e->kernel)
    if (int rc = check_kernel("spi_set_kernel_config", k.layout, min_blocks)) return rc;
  for (auto& k : e->kernel) k.min_blocks = min_blocks;
  if (e->graph_exec) { cudaGraphExecDestroy(e->graph_exec); e->graph_exec = nullptr; }
  return SPI_OK;
}

int spi_set_kernel_layout(spi_engine* e, int layout) {
  if (!e) return set_error(SPI_EINVAL, "null engine");
  int rc = check_kernel("spi_set_kernel_layout", layout, 3);
  if (rc || (rc = prepare_kernel("spi_set_kernel_layout", layout))) return rc;
  for (auto& k : e->kernel) {
    k.layout = layout;
    if (layout != SPI_LAYOUT_LANE && k.min_blocks < 3) k.min_blocks = 3;
  }
  if (e->graph_exec) { cudaGraphExecDestroy(e->graph_exec); e->graph_exec = nullptr; }
  return SPI_OK;
}

int spi_set_kernel_for(spi_engine* e, int population, int layout, int min_blocks) {
  if (!e) return set_error(SPI_EINVAL, "null engine");
  int rc = check_kernel("spi_set_kernel_for", layout, min_blocks);
  if (rc || (rc = prepare_kernel("spi_set_kernel_for", layout))) return rc;
  e->kernel[population != 0].layout = layout;
  e->kernel[population != 0].min_blocks = min_blocks;
  if (population && e->graph_exec) { cudaGraphExecDestroy(e->graph_exec); e->graph_exec = nullptr; }
  return SPI_OK;
}

int spi_set_cost(spi_engine* e, int mode, const float* sq_weights) {
  if (!e) return set_error(SPI_EINVAL, "null engine");
  if (mode != 0 && mode != 1) return set_error(SPI_EINVAL, "spi_set_cost: mode %d not 0/1", mode);
  e->cost_mode = mode;
  if (sq_weights) memcpy(e->sq_w, sq_weights, sizeof(e->sq_w));
  if (e->graph_exec) { cudaGraphExecDestroy(e->graph_exec); e->graph_exec = nullptr; }
  return SPI_OK;
}

int spi_run(spi_engine* e) { return run_impl(e, nullptr, e && e->population); }

int spi_run_population(spi_engine* e) { return run_impl(e, nullptr, true); }

int spi_evaluate(spi_engine* e, const float* theta, int N, float* comp, float* cost) {
  if (!e || !theta) return set_error(SPI_EINVAL, "spi_evaluate: null argument");
  if (N <= 0) return set_error(SPI_EINVAL, "spi_evaluate: N=%d must be > 0", N);
  if (e->W <= 0 || e->H <= 0) return set_error(SPI_ESTATE, "spi_evaluate before spi_load_windows");
  if (e->kernel[0].layout != SPI_LAYOUT_LANE) {
    int rc = spi_set_theta(e, theta, N);
    if (!rc) rc = run_impl(e, nullptr, false);
    return rc ? rc : spi_read_costs(e, comp, cost);
  }
  const int G = (e->W + 7) / 8;
  int rc = reserve_theta(e, N);
  if (rc) return rc;
  e->N = N;
  e->population = false;
  e->ran = false;
  if ((rc = reserve_run(e))) {
    // no room for the run: the batch is set all the same, as by spi_set_theta before a spi_run that finds none
    cudaMemcpyAsync(e->theta.p, theta, (size_t)N * SPI_THETA_DIM * 4, cudaMemcpyDeviceToDevice, e->stream);
    return rc;
  }
  const WinView win{e->init.f(), e->act.f(), e->tgt.f(), e->weight.f(), e->W, e->H};
  const EvalArgs a{win, theta, e->partial.f(), N, G, (unsigned long long*)e->bad.p};
  cudaError_t ce = eval_launch(e->host_model, e->kernel[0].min_blocks, e->sms, a, e->stream);
  if (ce != cudaSuccess) return cuda_error(ce, "spi_evaluate: rollout launch");
  const float* w = e->sq_w;
  finalize_evaluate<<<blocks_for(N, 128), 128, 0, e->stream>>>(e->partial.f(), N, G, e->norm, e->cost_mode, w[0], w[1],
                                                               w[2], w[3], w[4], w[5], theta, e->theta.f(), e->comp.f(),
                                                               e->cost.f(), comp, cost);
  ce = cudaGetLastError();
  if (ce != cudaSuccess) return cuda_error(ce, "spi_evaluate: finalize launch");
  e->ran = true;
  return SPI_OK;
}

int spi_run_trace(spi_engine* e, float* trace) {
  if (!trace) return set_error(SPI_EINVAL, "spi_run_trace: null trace");
  return run_impl(e, trace, false);
}

int spi_read_costs(spi_engine* e, float* comp, float* cost) {
  if (!e) return set_error(SPI_EINVAL, "null engine");
  if (!e->ran) return set_error(SPI_ESTATE, "spi_read_costs before spi_run");
  cudaError_t ce = cudaSuccess;
  if (comp) ce = cudaMemcpyAsync(comp, e->comp.p, (size_t)e->N * SPI_N_COMP * 4, cudaMemcpyDefault, e->stream);
  if (ce == cudaSuccess && cost) ce = cudaMemcpyAsync(cost, e->cost.p, (size_t)e->N * 4, cudaMemcpyDefault, e->stream);
  if (ce != cudaSuccess) return cuda_error(ce, "spi_read_costs");
  return SPI_OK;
}

int spi_read_theta(spi_engine* e, float* theta) {
  if (!e || !theta) return set_error(SPI_EINVAL, "spi_read_theta: null argument");
  if (e->N <= 0) return set_error(SPI_ESTATE, "spi_read_theta: no theta batch");
  cudaError_t ce = cudaMemcpyAsync(theta, e->theta.p, (size_t)e->N * SPI_THETA_DIM * 4, cudaMemcpyDefault, e->stream);
  return ce == cudaSuccess ? SPI_OK : cuda_error(ce, "spi_read_theta");
}

int spi_sync(spi_engine* e, int64_t* n_nonfinite) {
  if (!e) return set_error(SPI_EINVAL, "null engine");
  cudaError_t ce = cudaStreamSynchronize(e->stream);
  if (ce != cudaSuccess) return cuda_error(ce, "spi_sync");
  if (n_nonfinite) {
    unsigned long long v = 0;
    ce = cudaMemcpy(&v, e->bad.p, sizeof(v), cudaMemcpyDeviceToHost);
    if (ce != cudaSuccess) return cuda_error(ce, "spi_sync: read counter");
    *n_nonfinite = (int64_t)v;
  }
  return SPI_OK;
}

}  // extern "C"
