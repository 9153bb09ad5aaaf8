// Pieces shared by the expert GEMMs whose N operand is the tokens: the cut of an expert's rows
// into token tiles, the reads of an accumulator with the weight rows as lanes, the protocol with
// the all-to-all, and the tables of an epilogue that stores to peers.
#pragma once

#include <cuda_runtime.h>

#include "../core/ptx.cuh"
#include "../core/tcgen05.cuh"
#include "../core/wait.cuh"
#include "a2a_device.cuh"
#include "a2a_params.h"

namespace pplx {
namespace tok {

constexpr uint32_t kNoSignal = 0xffffffffu;
constexpr int kQueue = 512;  // arrival adds that wait for one fence

template <int kTokens>
struct PeerStage {
  unsigned long long row_off[kTokens];  // arena offset of each token's combine slot
  uint32_t token[kTokens];              // kNoSignal: none
  uint32_t group[kTokens];              // first rank of the token's DP group
  uint32_t q_token[kQueue];
  uint32_t q_group_units[kQueue];
};

// Token tile of an expert: the fewest tiles of at most `most`, all of one width.
__device__ __forceinline__ int token_tiles(int rows, int most) { return (rows + most - 1) / most; }
__device__ __forceinline__ int token_width(int rows, int tiles) {
  return (((rows + tiles - 1) / tiles) + 15) & ~15;
}

// 16 lanes x 16 columns: thread t receives columns 2 * (t % 4) and the next one of lane t / 4
// (r[0], r[1]) and of lane t / 4 + 8 (r[2], r[3]), then the same of the next eight columns.
__device__ __forceinline__ void tmem_ld_16x256b_x2(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7])
      : "r"(taddr));
}

// 32 lanes x 16 columns, as two of the above.
__device__ __forceinline__ void load_group(uint32_t taddr, uint32_t (&lo)[8], uint32_t (&hi)[8]) {
  tmem_ld_16x256b_x2(taddr, lo);
  tmem_ld_16x256b_x2(taddr + (16u << 16), hi);
}

// Stores four 8 x 8 blocks of 16-bit values (32 weight rows x 8 tokens) with the token as row:
// lane l gives the address of token l % 8 of block l / 8.
__device__ __forceinline__ void stmatrix_x4_trans(void* smem, uint32_t r0, uint32_t r1, uint32_t r2,
                                                  uint32_t r3) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(
                   tc::smem_u32(smem)),
               "r"(r0), "r"(r1), "r"(r2), "r"(r3)
               : "memory");
}

// The 128 threads of one of the two epilogue warp groups.
__device__ __forceinline__ void sync_group(int wg) {
  asm volatile("bar.sync %0, 128;" ::"r"(2 + wg) : "memory");
}

// Staging-fed forms: waits until the rows of tile `c` have landed, that is for the arrival
// counters of exactly the sources whose rows the tile covers.  `landed` remembers the sources
// of the current expert that were already waited for.  False: a wait ran out.
__device__ __forceinline__ bool wait_tile_sources(const A2AParams& p, int expert, int first_row,
                                                  int end_row, int parity, const uint32_t* src_rows,
                                                  uint32_t& landed) {
  const WaitCtx w{p.status, p.timeout_ns, static_cast<uint32_t>(p.rank)};
  const uint32_t* arrived = reinterpret_cast<const uint32_t*>(p.peer[p.rank] + p.off_arrived_e) +
                            (static_cast<size_t>(parity) * p.nle + expert) * p.world;
  const uint32_t r0 = static_cast<uint32_t>(first_row);
  const uint32_t r1 = static_cast<uint32_t>(end_row);
  uint32_t first = 0;
  bool waited = false, ok = true;
  for (int s = 0; s < p.world && ok; ++s) {
    uint32_t n;
    if (src_rows != nullptr) {
      n = src_rows[expert * p.world + s];
    } else {
      const uint32_t v = ptx::ld_relaxed_sys(
          reinterpret_cast<const uint32_t*>(p.peer[p.rank] + p.off_counts_all) +
          (static_cast<size_t>(parity) * p.world + s) * p.num_experts + p.rank * p.nle + expert);
      n = v > 1u ? v - 1u : 0u;
    }
    if (n > 0 && first < r1 && first + n > r0 && !((landed >> s) & 1u)) {
      uint32_t seen;
      ok = wait_until(arrived + s, PredGe{n}, seen, w, kPhaseFusedGemm, static_cast<uint32_t>(s), n);
      landed |= 1u << s;
      waited = true;
    }
    first += n;
  }
  if (ok && waited) ptx::fence_proxy_async();
  return ok;
}

// One fence, then the queued adds on the tokens' arrival counters (one warp).
template <int kTokens>
__device__ __forceinline__ void flush(const A2AParams& p, const PeerStage<kTokens>* st,
                                      uint32_t count, int lane) {
  ptx::fence_acq_rel_sys();
  for (uint32_t i = lane; i < count; i += 32) {
    const uint32_t grp = st->q_group_units[i] & 0xffu;
    const uint32_t units = st->q_group_units[i] >> 8;
    for (int r = 0; r < min(p.dp_size, 8); ++r) {
      ptx::red_add_relaxed_sys(
          reinterpret_cast<uint32_t*>(p.peer[grp + r] + p.off_comb_arrived) + st->q_token[i], units);
    }
  }
  __syncwarp();
}

}  // namespace tok
}  // namespace pplx
