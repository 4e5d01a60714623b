// Batched step kernels: many particle systems (cutting instances of uneven size) advanced
// together, one launch per phase of the step for all of them (mf_batch_*). The reference keeps
// its constants in __constant__ memory per translation unit (actions_gpu.cu:438-469,
// interactions_gpu.cu:423-459, tool_gpu.cu:20-27), one system per process; here every system's
// constants and buffers are one entry of a device array, and each block of a batched launch
// finds its system by the block's index and runs the same kernel body as the single-system
// kernel on that system's share of the grid. The arithmetic of every system is the
// single-system step's, bit for bit (same bodies, same force-sum tree per 256 particles).
#pragma once

#include "mf_mixed.cuh"

namespace mf {

// one system's step parameters and buffers (bound to one parity of its double buffer)
struct __align__(16) batch_entry {
  params P;
  dev_buffers D;
};

// the batch's block maps: cell scan, phases of 256 threads per block, pair sums, return map, PSE heat
enum : int { MAP_SCAN = 0, MAP_256, MAP_PAIR, MAP_PLASTIC, MAP_PSE, NUM_MAPS };

// one batched launch: entries of every system and first[k] = the first grid block of system k
// (n + 1 values, first[n] = the grid size)
struct batch_map {
  const batch_entry *e;
  const int *first;
  int n;
};

// The system of batched block vb (the largest k with first[k] <= vb), its entry copied into
// shared memory by the block's threads (16-byte words), and the block's index and count within
// it. A batched launch passes its own block index; the persistent kernel each phase block it
// takes.
__device__ __forceinline__ blk batch_block_at(const batch_map &M, batch_entry &s, int vb) {
  __shared__ int s_k;
  if (threadIdx.x == 0) {
    int lo = 0, hi = M.n - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(M.first + mid) <= vb) lo = mid;
      else hi = mid - 1;
    }
    s_k = lo;
  }
  __syncthreads();
  const int k = s_k;
  static_assert(sizeof(batch_entry) % 16 == 0, "entries are whole 16-byte words");
  const int4 *src = reinterpret_cast<const int4 *>(M.e + k);
  int4 *dst = reinterpret_cast<int4 *>(&s);
  for (int w = threadIdx.x; w < (int)(sizeof(batch_entry) / 16); w += blockDim.x) dst[w] = __ldg(src + w);
  __syncthreads();
  const int f0 = __ldg(M.first + k), f1 = __ldg(M.first + k + 1);
  return blk{vb - f0, f1 - f0};
}
__device__ __forceinline__ blk batch_block(const batch_map &M, batch_entry &s) {
  return batch_block_at(M, s, (int)blockIdx.x);
}

static __global__ void __launch_bounds__(SCAN_THREADS) kb_scan(batch_map M) {
  MF_PDL_WAIT();
  MF_PDL_TRIGGER();
  __shared__ batch_entry s;
  const blk b = batch_block(M, s);
  scan_body(s.D, s.P.N, 0, b);
}

static __global__ void __launch_bounds__(BLOCK) kb_scatter(batch_map M) {
  MF_PDL_WAIT();
  MF_PDL_TRIGGER();
  __shared__ batch_entry s;
  const blk b = batch_block(M, s);
  scatter_body(s.P.N, s.D, 0, b);
}

template <bool MIXED>
static __global__ void __launch_bounds__(BLOCK, 4) kb_reorder(batch_map M) {
  MF_PDL_WAIT();
  MF_PDL_TRIGGER();
  __shared__ batch_entry s;
  const blk b = batch_block(M, s);
  reorder_body<true, MIXED>(s.P, s.D, b);
}

// The pair kernels for a block size chosen by the batch's tuner. A batched kernel reads its
// system's parameters from shared memory instead of the constant bank, which costs registers:
// its launch bounds leave more room per thread than the single-system kernel's, so that it
// does not spill.
template <int BS>
static __global__ void __launch_bounds__(BS) kb_pair_fp64(batch_map M) {
  MF_PDL_WAIT();
  MF_PDL_TRIGGER();
  __shared__ batch_entry s;
  const blk b = batch_block(M, s);
  __shared__ unsigned s_list[pair64_shared<BS>::WORDS];
  switch (pair64_lanes(s.P.N)) {  // the system's own rule, so that its sums are its own context's
    case 4: pair_fp64_body<BS, 4>(s.P, s.D, b, s_list); break;
    case 2: pair_fp64_body<BS, 2>(s.P, s.D, b, s_list); break;
    default: pair_fp64_body<BS, 1>(s.P, s.D, b, s_list); break;
  }
}

// the mixed pair sums of a system's block, in the parts of the system's size, at one lane per particle
template <int BS>
__device__ __forceinline__ void pair_mixed_system(const params &P, const dev_buffers &D, blk b, unsigned *s_list) {
  switch (mixed_parts(P.N)) {
    case 4: pair_mixed_body<BS, 1, 4, false>(P, D, b, s_list); break;
    case 2: pair_mixed_body<BS, 1, 2, false>(P, D, b, s_list); break;
    default: pair_mixed_body<BS, 1, 1, false>(P, D, b, s_list); break;
  }
}

template <int BS>
static __global__ void __launch_bounds__(BS, 640 / BS) kb_pair_mixed(batch_map M) {
  MF_PDL_WAIT();
  MF_PDL_TRIGGER();
  __shared__ batch_entry s;
  const blk b = batch_block(M, s);
  __shared__ unsigned s_list[mixed_shared<BS>::WORDS];
  pair_mixed_system<BS>(s.P, s.D, b, s_list);
}

template <int BS>
static __global__ void __launch_bounds__(BS) kb_pse(batch_map M) {
  MF_PDL_WAIT();
  MF_PDL_TRIGGER();
  __shared__ batch_entry s;
  const blk b = batch_block(M, s);
  switch (pair64_lanes(s.P.N)) {
    case 4: pse_body<BS, 4>(s.P, s.D, b); break;
    case 2: pse_body<BS, 2>(s.P, s.D, b); break;
    default: pse_body<BS, 1>(s.P, s.D, b); break;
  }
}

template <int BS>
__device__ __forceinline__ void pse_mixed_system(const params &P, const dev_buffers &D, blk b) {
  switch (mixed_parts(P.N)) {
    case 4: pse_mixed_body<BS, 4>(P, D, b); break;
    case 2: pse_mixed_body<BS, 2>(P, D, b); break;
    default: pse_mixed_body<BS, 1>(P, D, b); break;
  }
}

template <int BS>
static __global__ void __launch_bounds__(BS) kb_pse_mixed(batch_map M) {
  MF_PDL_WAIT();
  MF_PDL_TRIGGER();
  __shared__ batch_entry s;
  const blk b = batch_block(M, s);
  pse_mixed_system<BS>(s.P, s.D, b);
}

static __global__ void __launch_bounds__(FINISH_BLOCK, 4) kb_finish(batch_map M) {
  MF_PDL_WAIT();
  MF_PDL_TRIGGER();
  __shared__ batch_entry s;
  const blk b = batch_block(M, s);
  __shared__ finish_stage s_in;
  finish_flat_body<true, false, false, true>(s.P, s.D, b, &s_in);
}

static __global__ void __launch_bounds__(BLOCK) kb_close(batch_map M) {
  MF_PDL_WAIT();
  MF_PDL_TRIGGER();
  __shared__ batch_entry s;
  __shared__ close_shared s_close;
  batch_block(M, s);
  close_step(s.P, s.D, finish_blocks(s.P.N), s_close);
}

template <bool PAIRED>
static __global__ void __launch_bounds__(BLOCK, 2) kb_plastic(batch_map M) {
  MF_PDL_WAIT();
  MF_PDL_TRIGGER();
  __shared__ batch_entry s;
  const blk b = batch_block(M, s);
  __shared__ close_shared s_close;
  plastic_body<PAIRED>(s.P, s.D, b, s_close);
}

}  // namespace mf
