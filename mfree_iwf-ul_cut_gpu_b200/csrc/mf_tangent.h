// The differentiable step's entry (mf_tangent.cu): what it needs of a context.
#pragma once

#include "mf_kernels.cuh"

namespace mf {
namespace tg {

// Device memory of the differentiable step (its size follows the particle count and the number of
// directions): up to KEEP_BYTES of it kept by the context between calls and freed with the context's
// particles, more only during a call.
struct workspace {
  void *mem = nullptr;
  size_t bytes = 0;
};

// Runs skip + window steps on dual numbers from the state `now`, on `stream`, one copy of the
// system per derivative direction: `params` lists them (0..5: A, B, n, C, m, mu; none: the
// values only). out_dmean: d(mean Fc), d(mean Ff) per direction. Returns an MF_ code; *cuda_err
// the CUDA error behind MF_ERR_CUDA / MF_ERR_NOMEM.
int run_mean_force(const params &P, const dev_buffers &ctx_buffers, const state_set &now, mf_tool_state tool,
                   int max_cell, cudaStream_t stream, workspace &ws, int skip_steps, int window_steps,
                   const int *directions, int n_directions, double out_mean[2], double *out_dmean, int *cuda_err);
void release(workspace &ws);

}  // namespace tg
}  // namespace mf
