// Device helpers shared by the kernels that take part in the all-to-all protocol.
#pragma once

#include "../core/wait.cuh"
#include "a2a_params.h"

namespace pplx {

// Clears the packed-mode flag set of `parity` (all threads of one block call it).
__device__ __forceinline__ void reset_packed_flags(const A2AParams& p, int parity) {
  uint32_t* all = reinterpret_cast<uint32_t*>(p.peer[p.rank] + p.off_counts_all) +
                  static_cast<size_t>(parity) * p.world * p.num_experts;
  for (int i = threadIdx.x; i < p.world * p.num_experts; i += blockDim.x) all[i] = 0;
  uint32_t* arrived_e = reinterpret_cast<uint32_t*>(p.peer[p.rank] + p.off_arrived_e) +
                        static_cast<size_t>(parity) * p.nle * p.world;
  for (int i = threadIdx.x; i < p.nle * p.world; i += blockDim.x) arrived_e[i] = 0;
}

// World of one rank, in a combine: tokens of the dispatch it belongs to.  (Dispatch number n,
// counted from 1 in comb_iter, had the parity of n - 1.)
__device__ __forceinline__ uint32_t last_dispatched(const A2AParams& p) {
  const uint4 state = __ldcg(reinterpret_cast<const uint4*>(p.iter));
  return (state.y & 1u) != 0u ? state.z : state.w;
}

// First step of a combine (all threads of one block call it): the dispatch that produced the
// rows has finished on this rank, so clear the flag set it used and move on to the other one.
// No peer can write this set again before it has seen counts of this rank's next dispatch.
__device__ __forceinline__ void finish_dispatch_round(const A2AParams& p) {
  const int tid = threadIdx.x;
  const int parity = static_cast<int>(ptx::ld_volatile(p.iter) & 1u);
  uint32_t* counts = reinterpret_cast<uint32_t*>(p.peer[p.rank] + p.off_counts) +
                     a2a_counts_index(p, parity, 0, 0);
  uint32_t* arrived =
      reinterpret_cast<uint32_t*>(p.peer[p.rank] + p.off_arrived) + parity * p.world;
  const int P = p.world * p.nle;
  for (int q = tid; q < P; q += blockDim.x) counts[q] = 0;
  if (tid < p.world) arrived[tid] = 0;
  reset_packed_flags(p, parity);
  __syncthreads();
  if (tid == 0) {
    const uint32_t done = *p.iter;
    // Exactly one dispatch must have started since the last combine.
    const uint32_t started = ptx::ld_volatile(p.comb_iter);
    if (started != done + 1u)
      report_failure(p.status, kOutOfOrder, kPhaseCombinePayload, 0, done + 1u, started, p.rank);
    *p.iter = done + 1u;
  }
}

}  // namespace pplx
