// Dispatch and combine of an object whose world is one rank: every token and every expert
// live on this GPU, so nothing has to be staged for, or announced to, anybody.
//
// The general kernels (dispatch.cu, combine.cu) send a row per (token, k) into a staging region
// and copy it out again, and combine does the same on the way back: at 4096 tokens of the
// DeepSeek-V3 shape that is three passes over 243 MB of rows and three over 470 MB of expert
// outputs where one is needed (215 + 274 us measured).  Here
//
//  * dispatch reads each token once, converts it to e4m3 once where asked to, and stores it
//    straight into its rows of out_expert_x.  The row of (token, k) is its rank among the
//    entries of the same expert in token order.  A block owns a contiguous range of
//    (token, 512-byte chunk) units, counts the experts of all earlier tokens in shared memory
//    and ranks its own entries against each other, so the blocks agree on every row without
//    exchanging anything, and a few tokens still spread over the whole chip;
//  * dispatch leaves (local expert, row) of every (token, k) in `row_of`, and combine gathers
//    the top-k rows of each token from expert_y itself and writes the weighted sum.
//
// Every form of dispatch leaves both directions of that table behind: `row_of` for combine, and
// (token, k) of every row in `row_src` for the peer-storing down projection (after the packed send
// the staging-fed up projection writes that one), so that either half of the fused path goes
// with the other half of the plain one.
//
// Both are bound by DRAM from a few hundred tokens on and by launch plus two dependent memory
// round trips below that.  DeepSeek-V3 shape, fp8 in, bf16 out, kernel times before and after:
// 4096 tokens 215 -> 58 us (272 MB) and 274 -> 110 us (529 MB); 128 tokens 14.2 -> 6.8 and
// 15.1 -> 6.9 us; 1 token 7.9 -> 5.8 and 6.9 -> 4.4 us.  (Writing the second row table and clearing
// what an earlier dispatch left has since added 0.1 us to the pass of one token.)
//
// Called as separate halves, dispatch stages each TOKEN once (the send half must be done with
// the caller's tensor) and the receive half spreads it to its rows; a counter of staged units
// says when the receive half may start, so the halves may be on different streams.  The packed
// send of the fused MoE layer stores rows at their final, expert-major staging slots like the
// general one, without the exchange of histograms.  Combine called as halves uses the general
// kernels, which find the rows through `row_of`.
#include <algorithm>

#include <cuda_runtime.h>

#include "../core/device_utils.cuh"
#include "../core/ptx.cuh"
#include "../core/utils.h"
#include "../core/wait.cuh"
#include "a2a_device.cuh"
#include "a2a_kernels.h"
#include "a2a_params.h"
#include "combine_device.cuh"
#include "quant_device.cuh"

namespace pplx {
namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kBlocksPerSm = kSingleRankBlocksPerSm;  // 64 registers per thread
constexpr int kMinEntries = 512;  // (token, k) entries whose rows a block knows at a time

enum Form : int {
  kDirect = 0,  // rows to out_expert_x
  kStage = 1,   // send half: tokens to the staging
  kPacked = 2,  // send half of the fused path: rows to expert-major staging slots
};

__device__ __forceinline__ void stamp(const A2AParams& p, int first, int last) {
  if (p.trace != nullptr && blockIdx.x == 0 && threadIdx.x == 0) {
    const uint64_t t = ptx::globaltimer_ns();
    for (int s = first; s <= last; ++s) p.trace[s] = t;
  }
}

__device__ __forceinline__ void stamp_block(const A2AParams& p, int first_slot) {
  if (p.trace != nullptr && threadIdx.x == 0 && blockIdx.x < kTraceBlocks)
    p.trace[first_slot + blockIdx.x] = ptx::globaltimer_ns();
}

__device__ __forceinline__ int token_count(const uint32_t* bound_m, int num_tokens, int max_tokens) {
  int m = num_tokens;
  if (bound_m != nullptr) m = min(m, static_cast<int>(__ldg(bound_m)));
  return min(m, max_tokens);
}

// Chunks of 32 vectors per token, and one more for scales that the caller passes in.
__host__ __device__ __forceinline__ int chunks_of(const A2AParams& p, bool quantize) {
  return ((p.hidden_bytes >> 4) + 31) / 32 + (p.scale_bytes > 0 && !quantize ? 1 : 0);
}

__host__ __device__ __forceinline__ int entry_cap(const A2AParams& p) {
  return p.topk > kMinEntries ? p.topk : kMinEntries;
}

// Adds the experts of entries [0, n) to a histogram in shared memory.
__device__ __forceinline__ void count_experts(const uint32_t* indices, int n, uint32_t E,
                                              uint32_t* hist) {
  auto add = [&](uint32_t e) {
    if (e < E) atomicAdd(&hist[e], 1u);
  };
  int done = 0;
  if ((reinterpret_cast<uintptr_t>(indices) & 15) == 0) {
    const int nv = n >> 2;
#pragma unroll 4
    for (int v = threadIdx.x; v < nv; v += kThreads) {
      const uint4 q = __ldg(reinterpret_cast<const uint4*>(indices) + v);
      add(q.x);
      add(q.y);
      add(q.z);
      add(q.w);
    }
    done = nv << 2;
  }
  for (int i = done + threadIdx.x; i < n; i += kThreads) add(__ldg(indices + i));
}

struct Smem {
  unsigned long long* off;  // [entries] where the row of an entry starts, kNoOffset: nowhere
  uint2* place;             // [entries] {local expert, row}
  uint32_t* expert;         // [entries] expert of each entry, padded to a multiple of four
  uint32_t* base;           // [E] entries of earlier tokens per expert
  uint32_t* first;          // [E] kPacked: first staging slot of each expert
  uint32_t* mine;           // [E] kPacked: rows this block stored per expert
};
constexpr unsigned long long kNoOffset = ~0ull;
constexpr uint32_t kScalesInside = 1u << 31;

__device__ __forceinline__ Smem carve(uint8_t* s, int entries, int E) {
  Smem m;
  m.off = reinterpret_cast<unsigned long long*>(s);
  m.place = reinterpret_cast<uint2*>(m.off + entries);
  m.expert = reinterpret_cast<uint32_t*>(m.place + entries);
  m.base = m.expert + round_up<int>(entries, 4);
  m.first = m.base + E;
  m.mine = m.first + E;
  return m;
}

template <int kForm, bool kQuant>
__global__ void __launch_bounds__(kThreads, kBlocksPerSm)
    single_dispatch_kernel(const __grid_constant__ DispatchArgs a) {
  extern __shared__ __align__(16) uint8_t dyn_smem[];
  const A2AParams& p = a.p;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int E = p.num_experts, topk = p.topk;
  const int entries = entry_cap(p);
  const Smem sm = carve(dyn_smem, entries, E);
  ptx::wait_for_previous_kernels();
  ptx::let_next_kernel_start();
  stamp(p, kTrDispatchStart, kTrDispatchStart);
  stamp_block(p, kTrBlockDispatchStart);

  const int m = token_count(a.bound_m, a.num_tokens, p.max_tokens);
  const int nvec = p.hidden_bytes >> 4;
  const int nscale = p.scale_bytes >> 2;
  const int payload_chunks = (nvec + 31) >> 5;
  const int chunks = chunks_of(p, kQuant);
  const int grid = static_cast<int>(gridDim.x), blk = static_cast<int>(blockIdx.x);
  // This block's units.  A packed row is announced by the block that stored it, so packed
  // ranges are whole tokens.
  const uint32_t total = static_cast<uint32_t>(m) * chunks;
  uint32_t u0, u1;
  if constexpr (kForm == kPacked) {
    u0 = static_cast<uint32_t>(static_cast<uint64_t>(m) * blk / grid) * chunks;
    u1 = static_cast<uint32_t>(static_cast<uint64_t>(m) * (blk + 1) / grid) * chunks;
  } else {
    u0 = static_cast<uint32_t>(static_cast<uint64_t>(total) * blk / grid);
    u1 = static_cast<uint32_t>(static_cast<uint64_t>(total) * (blk + 1) / grid);
  }
  const int t0 = static_cast<int>(u0 / chunks);
  const int t1 = u1 > u0 ? static_cast<int>((u1 - 1) / chunks) + 1 : t0;
  const bool last_block = blk == grid - 1;

  // The vectors of this warp's next unit; asked for before the rows are known.
  int4 lo{}, hi{};
  auto load = [&](uint32_t u) {
    if (u >= u1) return;
    const int i = static_cast<int>(u / chunks);
    const int c = static_cast<int>(u - static_cast<uint32_t>(i) * chunks);
    const int v = c * 32 + lane;
    if (c >= payload_chunks || v >= nvec) return;
    const uint8_t* row = a.x + static_cast<int64_t>(i) * a.x_stride_row;
    if constexpr (kQuant) {
      lo = ptx::ld_nc_v4(row + (static_cast<size_t>(v) << 5));
      hi = ptx::ld_nc_v4(row + (static_cast<size_t>(v) << 5) + 16);
    } else {
      lo = ptx::ld_nc_v4(row + (static_cast<size_t>(v) << 4));
    }
  };
  uint32_t u = u0 + warp;
  load(u);

  // {iter, comb_iter, dispatched[0], dispatched[1]}.  (This kernel's first block changes comb_iter,
  // which no other block uses, and the dispatched of its parity.)
  const uint4 state = __ldcg(reinterpret_cast<const uint4*>(p.iter));
  const int parity = static_cast<int>(state.x & 1u);
  const uint32_t dispatched_before = parity != 0 ? state.z : state.w;
  if (blk == 0 && tid == 0) {
    // A new round begins; dispatches started must equal combines finished.
    const uint32_t iter_now = state.x, started = state.y;
    if (started != iter_now)
      report_failure(p.status, kOutOfOrder, kPhaseDispatchCounts, 0, iter_now, started, p.rank);
    *p.comb_iter = started + 1u;
    p.dispatched[parity] = static_cast<uint32_t>(m);
    if constexpr (kForm == kStage) {
      // Tokens staged by this half, + 1, and whether their scales come with their payload: the
      // receive half may be a call of the other kind.  (Rows per expert travel in recv_count.)
      ptx::st_relaxed_sys(reinterpret_cast<uint32_t*>(p.peer[p.rank] + p.off_counts) +
                              a2a_counts_index(p, parity, 0, 0),
                          static_cast<uint32_t>(m) + 1u | (kQuant ? kScalesInside : 0u));
    }
  }
  for (int e = tid; e < E; e += kThreads) {
    sm.base[e] = 0;
    if constexpr (kForm == kPacked) {
      sm.first[e] = 0;
      sm.mine[e] = 0;
    }
  }
  __syncthreads();
  count_experts(a.indices, t0 * topk, E, sm.base);
  if constexpr (kForm == kPacked) {
    // Slots are expert-major: this form needs the totals of all tokens as well.
    __syncthreads();
    count_experts(a.indices + static_cast<size_t>(t0) * topk, (m - t0) * topk, E, sm.first);
    __syncthreads();
    for (int e = tid; e < E; e += kThreads) sm.first[e] += sm.base[e];
    __syncthreads();
    if (blk == 0) {
      uint32_t* all = reinterpret_cast<uint32_t*>(p.peer[p.rank] + p.off_counts_all) +
                      static_cast<size_t>(parity) * E;
      for (int e = tid; e < E; e += kThreads) ptx::st_relaxed_sys(all + e, sm.first[e] + 1u);
      __syncthreads();
    }
    if (warp == 0) warp_exclusive_scan_smem(sm.first, E, lane, false);
  }
  __syncthreads();
  stamp(p, kTrDispatchHist, kTrDispatchHist);

  const int batch_tokens = max(1, entries / topk);
  for (int tb = t0; tb < t1; tb += batch_tokens) {
    const int te = min(tb + batch_tokens, t1);
    const int n = (te - tb) * topk;
    for (int j = tid; j < round_up<int>(n, 4); j += kThreads)
      sm.expert[j] =
          j < n ? __ldg(a.indices + static_cast<size_t>(tb) * topk + j) : 0xffffffffu;
    __syncthreads();
    for (int j = tid; j < n; j += kThreads) {
      const uint32_t e = sm.expert[j];
      const int i = tb + j / topk;
      // The block that moves a token's first chunk also writes its places down.
      const bool owner = static_cast<uint32_t>(i) * chunks >= u0;
      uint2 place = make_uint2(kNoRow, 0u);
      unsigned long long off = kNoOffset;
      if (e < static_cast<uint32_t>(E)) {
        uint32_t row = sm.base[e];
        const uint4* seen = reinterpret_cast<const uint4*>(sm.expert);
        for (int v = 0; v < (j >> 2); ++v) {
          const uint4 q = seen[v];
          row += (q.x == e) + (q.y == e) + (q.z == e) + (q.w == e);
        }
        for (int v = j & ~3; v < j; ++v) row += sm.expert[v] == e;
        if constexpr (kForm == kPacked) {
          const uint32_t pos = sm.first[e] + row;
          if (pos < static_cast<uint32_t>(p.region_slots)) {
            place = make_uint2(e, row);
            off = static_cast<unsigned long long>(pos) * p.slot_bytes;
            atomicAdd(&sm.mine[e], 1u);
          } else if (owner) {
            report_failure(p.status, kSlotOverflow, kPhaseDispatchPayload, 0, p.region_slots, pos,
                           p.rank);
          }
        } else {
          // Only a token that names one expert twice can run past the capacity.
          if (row < static_cast<uint32_t>(p.cap)) {
            place = make_uint2(e, row);
            off = e * static_cast<unsigned long long>(a.out_x_stride_e) +
                  row * static_cast<unsigned long long>(a.out_x_stride_row);
          } else if (owner) {
            report_failure(p.status, kRowOverflow, kPhaseDispatchPayload, 0, p.cap, row, p.rank);
          }
        }
      } else if (p.debug_checks && owner) {
        report_failure(p.status, kBadExpert, kPhaseDispatchCounts, i, E, e, p.rank);
      }
      if constexpr (kForm != kStage) {
        sm.place[j] = place;
        sm.off[j] = off;
      }
      if (owner) {
        uint2 kept = place;
        if constexpr (kForm == kPacked) {
          // (The slot exists, but expert_y has no row for it.)
          if (place.y >= static_cast<uint32_t>(p.cap)) kept = make_uint2(kNoRow, 0u);
        } else if (place.x != kNoRow) {
          p.row_src[static_cast<size_t>(e) * p.cap + place.y] =
              make_uint2(static_cast<uint32_t>(p.rank) | static_cast<uint32_t>(j - (i - tb) * topk) << 16,
                         static_cast<uint32_t>(i));
        }
        p.row_of[static_cast<size_t>(tb) * topk + j] = kept;
      }
    }
    __syncthreads();
    if (tb == t0) stamp(p, kTrDispatchPosted, kTrDispatchPosted);

    const uint32_t u_end = min(u1, static_cast<uint32_t>(te) * chunks);
    while (u < u_end) {
      const int i = static_cast<int>(u / chunks);
      const int c = static_cast<int>(u - static_cast<uint32_t>(i) * chunks);
      const int v = c * 32 + lane;
      const int j0 = (i - tb) * topk;
      const int4 cur_lo = lo, cur_hi = hi;
      u += kWarps;
      load(u);
      if (c < payload_chunks) {
        const bool live = v < nvec;
        int4 out = cur_lo;
        float scale = 0.f;
        if constexpr (kQuant) warp_quantize16(cur_lo, cur_hi, live, p.quant_pow2 != 0, out, scale);
        if (live) {
          if constexpr (kForm == kStage) {
            uint8_t* slot = p.peer[p.rank] + p.off_disp_stage + static_cast<size_t>(i) * p.slot_bytes;
            ptx::st_v4(slot + (static_cast<size_t>(v) << 4), out);
            if (kQuant && (lane & 7) == 0)
              reinterpret_cast<float*>(slot + p.hidden_bytes)[v >> 3] = scale;
          } else {
            uint8_t* dst = kForm == kPacked ? p.peer[p.rank] + p.off_disp_stage : a.out_x;
            dst += static_cast<size_t>(v) << 4;
#pragma unroll 4
            for (int k = 0; k < topk; ++k) {
              const unsigned long long off = sm.off[j0 + k];
              if (off != kNoOffset) ptx::st_v4(dst + off, out);
            }
            if (kQuant && (lane & 7) == 0) {
              for (int k = 0; k < topk; ++k) {
                const uint2 place = sm.place[j0 + k];
                if (place.x == kNoRow) continue;
                if constexpr (kForm == kPacked) {
                  reinterpret_cast<float*>(p.peer[p.rank] + p.off_disp_stage + sm.off[j0 + k] +
                                           p.hidden_bytes)[v >> 3] = scale;
                } else {
                  a.out_scale[place.x * a.out_scale_stride_e + place.y * a.out_scale_stride_row +
                              (v >> 3) * a.out_scale_stride_col] = scale;
                }
              }
            }
          }
        }
        if (kForm == kPacked && c == 0) {
          for (int k = lane; k < topk; k += 32) {
            if (sm.off[j0 + k] != kNoOffset)
              ptx::st_v4(p.peer[p.rank] + p.off_disp_stage + sm.off[j0 + k] + p.trailer_off,
                         make_int4(i, k, static_cast<int>(sm.place[j0 + k].x), p.rank));
          }
        }
      } else {
        // The scales that came with the token.
        const float* src = a.x_scale + static_cast<int64_t>(i) * a.x_scale_stride_row;
        for (int s = lane; s < nscale; s += 32) {
          const float scale = __ldg(src + s * a.x_scale_stride_col);
          if constexpr (kForm == kStage) {
            reinterpret_cast<float*>(p.peer[p.rank] + p.off_disp_stage +
                                     static_cast<size_t>(i) * p.slot_bytes + p.hidden_bytes)[s] = scale;
          } else {
#pragma unroll 4
            for (int k = 0; k < topk; ++k) {
              const uint2 place = sm.place[j0 + k];
              if (place.x != kNoRow)
                a.out_scale[place.x * a.out_scale_stride_e + place.y * a.out_scale_stride_row +
                            s * a.out_scale_stride_col] = scale;
            }
          }
        }
      }
    }
    // The next batch's entries come after these.
    __syncthreads();
    if (last_block || te < t1) {
      for (int j = tid; j < n; j += kThreads) {
        const uint32_t e = sm.expert[j];
        if (e < static_cast<uint32_t>(E)) atomicAdd(&sm.base[e], 1u);
      }
      __syncthreads();
    }
  }
  if (last_block) {
    // Tokens that the dispatch before had and this one does not.
    for (uint32_t j = static_cast<uint32_t>(m) * topk + tid; j < dispatched_before * topk; j += kThreads)
      p.row_of[j] = make_uint2(kNoRow, 0u);
  }
  stamp(p, kTrDispatchStored, kTrDispatchStored);

  if constexpr (kForm == kPacked) {
    // (The loop above ended with a block barrier.)  One fence for the block, then one relaxed
    // add per expert that got rows.
    if (warp == 0 && t1 > t0) {
      ptx::fence_acq_rel_gpu();
      for (int e = lane; e < E; e += 32) {
        const uint32_t n = sm.mine[e];
        if (n != 0)
          ptx::red_add_relaxed_sys(reinterpret_cast<uint32_t*>(p.peer[p.rank] + p.off_arrived_e) +
                                       static_cast<size_t>(parity) * p.nle + e,
                                   n);
      }
    }
  } else if (last_block) {
    // No token follows the last block's: its counts are the totals.
    for (int e = tid; e < E; e += kThreads) {
      if constexpr (kForm == kDirect) a.out_num_tokens[e] = static_cast<int32_t>(sm.base[e]);
      else p.recv_total[e] = sm.base[e];
      p.recv_count[e] = min(sm.base[e], static_cast<uint32_t>(p.cap));
    }
  }
  if constexpr (kForm == kStage) {
    __syncthreads();
    // One unit more for the last block, for its totals, and one for the first, for the state of the
    // object: both are announced even when there is no token.
    const uint32_t more = (last_block ? 1u : 0u) + (blk == 0 ? 1u : 0u);
    if (tid == 0 && (u1 - u0) + more > 0)
      ptx::red_add_release_gpu(
          reinterpret_cast<uint32_t*>(p.peer[p.rank] + p.off_arrived) + parity, (u1 - u0) + more);
  }
  stamp(p, kTrDispatchSignalled, kTrDispatchEnd);
  stamp_block(p, kTrBlockDispatchEnd);
}

// Receive half: staged tokens to their rows.
__global__ void __launch_bounds__(kThreads, kBlocksPerSm)
    single_unstage_kernel(const __grid_constant__ DispatchArgs a) {
  __shared__ uint32_t s_tokens;
  const A2AParams& p = a.p;
  ptx::wait_for_previous_kernels();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int topk = p.topk;
  const int nvec = p.hidden_bytes >> 4;
  const int nscale = p.scale_bytes >> 2;
  const int payload_chunks = (nvec + 31) >> 5;
  const int chunks = payload_chunks + (nscale > 0 ? 1 : 0);
  const int parity = static_cast<int>(ptx::ld_volatile(p.iter) & 1u);
  if (tid == 0) {
    const WaitCtx w{p.status, p.timeout_ns, static_cast<uint32_t>(p.rank)};
    uint32_t v = 0, seen = 0;
    bool ok = wait_until(reinterpret_cast<const uint32_t*>(p.peer[p.rank] + p.off_counts) +
                             a2a_counts_index(p, parity, 0, 0),
                         PredNonZero{}, v, w, kPhaseDispatchCounts, p.rank, 1u);
    const uint32_t sent = (v & kScalesInside) != 0u ? payload_chunks : chunks;
    v &= ~kScalesInside;
    const uint32_t units = ok ? (v - 1u) * sent + 2u : 0u;
    ok = ok && wait_until(reinterpret_cast<const uint32_t*>(p.peer[p.rank] + p.off_arrived) + parity,
                          PredGe{units}, seen, w, kPhaseDispatchPayload, p.rank, units);
    s_tokens = ok ? v - 1u : 0u;
  }
  __syncthreads();
  stamp(p, kTrDispatchCounts, kTrDispatchLayout);
  if (blockIdx.x == 0) {
    for (int e = tid; e < p.nle; e += kThreads)
      a.out_num_tokens[e] = static_cast<int32_t>(__ldcg(p.recv_total + e));
  }
  const uint32_t total = s_tokens * chunks;
  const uint8_t* stage = p.peer[p.rank] + p.off_disp_stage;
  for (uint32_t u = blockIdx.x * kWarps + warp; u < total; u += gridDim.x * kWarps) {
    const int i = static_cast<int>(u / chunks);
    const int c = static_cast<int>(u - static_cast<uint32_t>(i) * chunks);
    const uint8_t* slot = stage + static_cast<size_t>(i) * p.slot_bytes;
    const uint2* places = p.row_of + static_cast<size_t>(i) * topk;
    if (c < payload_chunks) {
      const int v = c * 32 + lane;
      if (v >= nvec) continue;
      const int4 r = ptx::ld_cg_v4(slot + (static_cast<size_t>(v) << 4));
#pragma unroll 8
      for (int k = 0; k < topk; ++k) {
        const uint2 place = __ldcg(places + k);
        if (place.x != kNoRow)
          ptx::st_v4(a.out_x + place.x * a.out_x_stride_e + place.y * a.out_x_stride_row +
                         (static_cast<size_t>(v) << 4),
                     r);
      }
    } else {
      for (int s = lane; s < nscale; s += 32) {
        const float scale = __ldcg(reinterpret_cast<const float*>(slot + p.hidden_bytes) + s);
#pragma unroll 4
        for (int k = 0; k < topk; ++k) {
          const uint2 place = __ldcg(places + k);
          if (place.x != kNoRow)
            a.out_scale[place.x * a.out_scale_stride_e + place.y * a.out_scale_stride_row +
                        s * a.out_scale_stride_col] = scale;
        }
      }
    }
  }
  stamp(p, kTrDispatchCopied, kTrDispatchEnd);
}

// Combine: the top-k rows of each token, gathered from expert_y and summed in k order.  A warp
// unit is kVec vectors per lane of one token; all loads of up to kBatch rows are in flight at
// once, and where they are is looked up one unit ahead (lane k holds row and weight k).
template <typename T, typename U, int kVec>
__global__ void __launch_bounds__(kThreads, kBlocksPerSm)
    single_combine_kernel(const __grid_constant__ CombineArgs a) {
  const A2AParams& p = a.p;
  ptx::wait_for_previous_kernels();
  ptx::let_next_kernel_start();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m = token_count(a.bound_m, a.num_tokens, p.max_tokens);
  const int topk = p.topk;
  const int nvec8 = p.hidden_dim >> 3;
  const uint32_t chunks = static_cast<uint32_t>((nvec8 + 32 * kVec - 1) / (32 * kVec));
  const uint32_t total = static_cast<uint32_t>(m) * chunks;
  const uint32_t gwarps = gridDim.x * kWarps;
  stamp(p, kTrCombineStart, kTrCombineSent);
  stamp_block(p, kTrBlockCombineStart);

  uint2 place{kNoRow, 0};
  float weight = 0.f;
  auto look_up = [&](uint32_t u, int k0) {
    place = make_uint2(kNoRow, 0);
    if (u >= total || k0 + lane >= topk) return;
    const size_t i = u / chunks;
    place = __ldg(p.row_of + i * topk + k0 + lane);
    weight = __ldg(a.weights + static_cast<int64_t>(i) * a.w_stride_row + k0 + lane);
  };
  uint32_t u = blockIdx.x * kWarps + warp;
  look_up(u, 0);

  // The per-token arrival counters of the staged forms stay in step (see recv_phase_ll).
  {
    uint32_t* arrived = reinterpret_cast<uint32_t*>(p.peer[p.rank] + p.off_comb_arrived);
    const uint32_t per_round = static_cast<uint32_t>(topk) * static_cast<uint32_t>(p.comb_units);
    for (int i = blockIdx.x * kThreads + tid; i < p.max_tokens; i += gridDim.x * kThreads)
      atomicAdd(arrived + i, per_round);
  }
  if (blockIdx.x == gridDim.x - 1) finish_dispatch_round(p);

  const T* y = static_cast<const T*>(a.expert_y);
  U* out = static_cast<U*>(a.out_tokens);
  constexpr int kBatch = (sizeof(T) == 4 ? 4 : 8) / kVec;
  for (; u < total; u += gwarps) {
    const int i = static_cast<int>(u / chunks);
    const int v0 = static_cast<int>(u - static_cast<uint32_t>(i) * chunks) * 32 * kVec + lane;
    float acc[kVec][8];
#pragma unroll
    for (int q = 0; q < kVec; ++q) {
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[q][j] = 0.f;
    }
    bool whole = true;
    for (int k0 = 0; k0 < topk; k0 += kBatch) {
      if (k0 > 0 && (k0 & 31) == 0) look_up(u, k0);
      Vec8<T> x[kVec][kBatch];
      float w[kBatch];
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        const int src = (k0 + j) & 31;
        const uint32_t le = __shfl_sync(0xffffffffu, place.x, src);
        const uint32_t row = __shfl_sync(0xffffffffu, place.y, src);
        w[j] = __shfl_sync(0xffffffffu, weight, src);
        if (k0 + j < topk) {
          if (le == kNoRow) {
            whole = false;
          } else {
            const T* base = y + le * a.y_stride_e + row * a.y_stride_row;
#pragma unroll
            for (int q = 0; q < kVec; ++q) {
              if (v0 + 32 * q < nvec8) x[q][j].load_nc(base + static_cast<int64_t>(v0 + 32 * q) * 8);
            }
          }
        }
      }
      if (k0 + kBatch >= topk) look_up(u + gwarps, 0);
      if (!whole) continue;
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        if (k0 + j < topk) {
#pragma unroll
          for (int q = 0; q < kVec; ++q) x[q][j].fma_into(acc[q], w[j]);
        }
      }
    }
    if (!whole) {
      // The token was not dispatched, or an entry of it named no expert: it has no result.
      if (lane == 0) {
        const uint32_t had = last_dispatched(p);
        const bool known = static_cast<uint32_t>(i) < had;
        report_failure(p.status, known ? kBadExpert : kBadToken, kPhaseCombinePayload, i,
                       known ? topk : had, known ? 0 : i, p.rank);
      }
      continue;
    }
#pragma unroll
    for (int q = 0; q < kVec; ++q) {
      if (v0 + 32 * q < nvec8)
        ptx::st_v4(out + static_cast<int64_t>(i) * a.out_stride_row +
                       static_cast<int64_t>(v0 + 32 * q) * 8,
                   pack8(acc[q], static_cast<U*>(nullptr)));
    }
  }
  stamp(p, kTrCombineReduced, kTrCombineEnd);
  stamp_block(p, kTrBlockCombineEnd);
}

size_t dispatch_smem(const A2AParams& p) {
  const size_t n = entry_cap(p);
  return n * 16 + sizeof(uint32_t) * (round_up<size_t>(n, 4) + 3 * static_cast<size_t>(p.num_experts));
}

int grid_for(int64_t units, int limit) {
  return static_cast<int>(std::clamp<int64_t>((units + kWarps - 1) / kWarps, 1, limit));
}

cudaError_t launch(const void* fn, int grid, size_t smem, void** params, cudaStream_t stream) {
  if (smem > 48 * 1024) {
    const cudaError_t err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 static_cast<int>(smem));
    if (err != cudaSuccess) return err;
  }
  return launch_after_previous(fn, dim3(grid), dim3(kThreads), params, smem, stream);
}

}  // namespace

size_t single_rank_smem_bytes(const A2AParams& p) { return dispatch_smem(p); }

cudaError_t launch_single_dispatch(const DispatchArgs& a, bool send, bool recv, int one_per_sm,
                                   int limit, cudaStream_t stream) {
  const bool quant = a.quantize != 0;
  const int64_t units = static_cast<int64_t>(a.num_tokens) * chunks_of(a.p, quant);
  if (!send) {
    void* params[] = {const_cast<DispatchArgs*>(&a)};
    return launch(reinterpret_cast<const void*>(&single_unstage_kernel), grid_for(units, one_per_sm), 0,
                  params, stream);
  }
  const void* fn;
  if (a.packed) {
    fn = quant ? reinterpret_cast<const void*>(&single_dispatch_kernel<kPacked, true>)
               : reinterpret_cast<const void*>(&single_dispatch_kernel<kPacked, false>);
  } else if (recv) {
    fn = quant ? reinterpret_cast<const void*>(&single_dispatch_kernel<kDirect, true>)
               : reinterpret_cast<const void*>(&single_dispatch_kernel<kDirect, false>);
  } else {
    fn = quant ? reinterpret_cast<const void*>(&single_dispatch_kernel<kStage, true>)
               : reinterpret_cast<const void*>(&single_dispatch_kernel<kStage, false>);
  }
  void* params[] = {const_cast<DispatchArgs*>(&a)};
  // (Staging stores a chunk once, not top-k times: twice the blocks only count twice.)
  const int grid = a.packed ? std::clamp(a.num_tokens, 1, one_per_sm)
                            : grid_for(units, recv ? limit : one_per_sm);
  return launch(fn, grid, dispatch_smem(a.p), params, stream);
}

cudaError_t launch_single_combine(const CombineArgs& a, DType in, DType out, int limit,
                                  cudaStream_t stream) {
  const int vecs = ((a.p.hidden_dim >> 3) + 31) / 32;
  // Two vectors per lane where a token has few rows and there are enough tokens to keep every
  // warp at work all the same: with top-2 one vector is two 16-byte loads in flight per lane.
  const bool pairs = a.p.topk <= 4 && static_cast<int64_t>(a.num_tokens) * vecs >= 2 * kWarps * limit;
  const int64_t units = static_cast<int64_t>(a.num_tokens) * (pairs ? (vecs + 1) / 2 : vecs);
  const int grid = grid_for(units, limit);
  return dispatch_types(in, out, [&]<typename T, typename U>() {
    void* params[] = {const_cast<CombineArgs*>(&a)};
    const void* fn = pairs ? reinterpret_cast<const void*>(&single_combine_kernel<T, U, 2>)
                           : reinterpret_cast<const void*>(&single_combine_kernel<T, U, 1>);
    return launch(fn, grid, 0, params, stream);
  });
}

}  // namespace pplx
