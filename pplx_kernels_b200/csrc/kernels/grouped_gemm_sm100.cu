// Grouped expert GEMM for sm_100a: for every local expert e with counts[e] rows,
//   out[e, :counts[e], :] = act(x[e, :counts[e], :] @ w[e]^T)
// with bf16 operands, fp32 accumulation in tensor memory and a bf16 result.
// `act` is the identity, or SwiGLU when w[e] stacks a gate and an up projection
// ([2 * I, K]) and the result has I columns: silu(x @ gate^T) * (x @ up^T).
//
// The reference contains no GEMM; this kernel serves the fused MoE layer that
// goes beyond it.
//
// The WEIGHTS are the M operand of the MMAs and the tokens the N operand.  A CTA pair
// (tcgen05 cta_group::2) owns a tile of 256 weight rows, 128 in each CTA's tensor-memory
// lanes, times a token tile of 32 to 512 rows of one expert in steps of 32; each CTA loads its
// own weight rows and HALF of the tokens, and the leader's MMAs read both CTAs' shared
// memory.  An expert's rows are cut into equal token tiles (to a step), so
//   - weights cross from DRAM once and from L2 once for up to 512 rows of an expert (two MMAs per
//     step above 256),
//   - the work follows the rows there are, to a multiple of 32: with the tokens as M every
//     expert was padded to a multiple of 128 rows (256 for pairs, which therefore were only
//     used from 2048 rows per expert on),
//   - a pair reads 64 bytes per SM and clock from L2 at the full MMA rate; one CTA per
//     128 x 256 tile needs 96, and L2 delivers about 64: that bound the kernel at 1.0 PFLOP/s.
// The SwiGLU form interleaves eight gate rows with eight up rows in shared memory (a
// five-dimensional tensor map does that on the way), so that the 16x256b reads of tensor memory
// give a thread both halves of its results.
//
// Layers before and after: Mixtral 8x7B (8 experts of 14336 x 4096) with 512 tokens 647 -> 543 us
// and with 4096 tokens 2867 -> 2640 us, Qwen3-30B-A3B (128 experts of 768 x 2048) with 16 tokens
// 191 -> 158 us.
//
// Roles (persistent over tiles): warp 0 TMA producer, warp 1 MMA issuer (leader CTA only),
// warp 2 tensor-memory allocation, warps 4-11 epilogue.  Two accumulators of 256 columns let
// the epilogue of a tile run under the MMAs of the next; wider tiles have one of 512 columns.  No TMA multicast is involved: the two
// CTAs load different data; only barrier arrivals (tcgen05.commit) are delivered to both.
//
// Tiles are (expert, block of weight rows, token tile) with the token tile varying fastest, so
// CTAs that run at the same time share weights in L2.  The row counts are read on the device,
// so the launch is graph-capturable and does no work for empty experts.
//
// Two template switches turn the same pipeline into the compute+collective
// kernels of the fused MoE layer:
//
//   kFromStaging   the tokens are read by TMA straight out of the dispatch
//                  staging arena that PEERS fill with P2P stores (packed send:
//                  rows grouped by local expert, then by source rank, dense).
//                  Arrival is counted per (expert, source): before a tile the
//                  producer warp waits (ld.acquire.sys, then fence.proxy.async)
//                  only for the sources whose rows the tile covers, so the expert
//                  GEMM starts tile by tile as tokens land and the receive-side
//                  copy of dispatch disappears.  The epilogue also records
//                  (source, token, k) of every row for combine.
//   kToPeers       the epilogue does not write a local result: every output row
//                  is stored into the combine staging of the token's home rank(s)
//                  over NVLink in 256-byte pieces, followed by a system-scope fence
//                  per handful of tiles and relaxed adds on the tokens' arrival counters.
//                  The combine send kernel and the expert_y round trip disappear.
//
// Every mbarrier wait is bounded: when one runs out the CTA raises a shared
// abort flag, all roles leave their loops, in-flight TMA loads are drained,
// tensor memory is freed and the kernel returns with *status = 1.
#include <algorithm>

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../core/device_utils.cuh"
#include "../core/ptx.cuh"
#include "../core/tcgen05.cuh"
#include "../core/utils.h"
#include "../core/wait.cuh"
#include "a2a_device.cuh"
#include "grouped_gemm.h"
#include "token_tile.cuh"

namespace pplx {
namespace {

using namespace tok;

constexpr int kBlockM = 128;      // weight rows per CTA and tile
constexpr int kMmaTokens = 256;   // token rows per MMA
constexpr int kMaxTokens = 512;   // token rows per tile
constexpr int kBlockK = 64;       // 64 bf16 = one 128-byte swizzle row
constexpr int kUmmaK = 16;
constexpr int kMaxStages = 12;
constexpr int kThreads = 384;
constexpr int kTmemCols = 512;    // an accumulator of kMaxTokens columns, or two of half of them
constexpr uint32_t kRowBytes = kBlockK * 2;
constexpr uint32_t kWBytes = kBlockM * kRowBytes;
constexpr uint32_t kWaitLimitNs = 2000000000u;  // 2 s per wait
constexpr int kMaxExperts = 1024;
constexpr int kDrainPlain = 8;    // cycles per token row to read out an accumulator that is the only
constexpr int kDrainSwiglu = 35;  // one, as fitted to the times of both widths at 512 rows
constexpr int kSegBytes = 256 + 16;  // 128 bf16 columns of one token, padded

struct Control {
  uint64_t full[kMaxStages];
  uint64_t empty[kMaxStages];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint32_t tmem_base;
  uint32_t abort_flag;
  uint32_t max_rows;                // rows of the largest expert
  uint32_t max_width;               // widest token tile of this launch
  unsigned long long best_limit;    // (cost << 16) | limit of the token tile
  alignas(16) uint8_t seg[2][2][16][kSegBytes];  // [warp group][alternating][token][column]
};

// Token rows come in boxes of 64 and 16.
struct TokenMaps {
  CUtensorMap x64, x16;
};

struct Tile {
  int expert;
  int w_blk;    // block of weight rows (of the pair or the single CTA)
  int first;    // first token row of the tile inside its expert
  int width;    // token rows of the tile, a multiple of kUnit
  int rows;     // valid rows of the expert
};

// Token tiles of an expert: as few as `limit` rows per tile allow, as equal as whole units allow.
template <int kUnit>
struct Cut {
  int units, tiles;
  __device__ __forceinline__ Cut(int rows, int limit)
      : units((rows + kUnit - 1) / kUnit), tiles((units * kUnit + limit - 1) / limit) {}
  __device__ __forceinline__ int widest() const { return (units + tiles - 1) / tiles * kUnit; }
};

template <int kUnit>
__device__ __forceinline__ Tile locate(const uint32_t* tile_start, const uint32_t* rows_of,
                                       int num_experts, int limit, uint32_t t) {
  Tile c;
  c.expert = find_group(tile_start, num_experts, t);
  c.rows = static_cast<int>(rows_of[c.expert]);
  const Cut<kUnit> cut(c.rows, limit);
  const uint32_t rem = t - tile_start[c.expert];
  c.w_blk = static_cast<int>(rem / cut.tiles);
  const int i = static_cast<int>(rem) - c.w_blk * cut.tiles;
  const int each = cut.units / cut.tiles, wider = cut.units - each * cut.tiles;
  c.width = (each + (i < wider ? 1 : 0)) * kUnit;
  c.first = (i * each + min(i, wider)) * kUnit;
  return c;
}

__device__ __forceinline__ float silu(float v) { return v / (1.0f + __expf(-v)); }

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ uint32_t pack_bits(uint32_t a, uint32_t b) {
  return pack_bf16(__uint_as_float(a), __uint_as_float(b));
}

// Two tokens' results of one column from their gate and up sums.
__device__ __forceinline__ uint32_t swiglu_pair(uint32_t g0, uint32_t g1, uint32_t u0, uint32_t u1) {
  return pack_bf16(silu(__uint_as_float(g0)) * __uint_as_float(u0),
                   silu(__uint_as_float(g1)) * __uint_as_float(u1));
}

// Token rows of a tile that its first MMA takes; the second takes the rest.
__device__ __forceinline__ int first_mma(int width) {
  return width <= kMmaTokens ? width : ((width >> 1) + 31) & ~31;
}

template <bool kPair>
__device__ __forceinline__ void load_rows(void* dst, const CUtensorMap* map, uint64_t* full, int k,
                                          int row, int plane) {
  if constexpr (kPair) tc::tma_load_3d_2cta(dst, map, full, k, row, plane);
  else tc::tma_load_3d(dst, map, full, k, row, plane);
}

template <bool SWIGLU, bool kFromStaging, bool kToPeers, bool kPair, bool kWide>
__global__ void __launch_bounds__(kThreads, 1)
    grouped_gemm_kernel(const __grid_constant__ CUtensorMap tmap_w,
                        const __grid_constant__ TokenMaps tmap_x,
                        const __grid_constant__ GroupedGemmArgs g) {
  static_assert(kPair || !kWide, "one CTA has no room for the stages of wide tiles");
  constexpr int kCtas = kPair ? 2 : 1;
  constexpr int kUnit = 16 * kCtas;  // steps of an MMA's N: 16, or 32 for M = 256 over a pair
  constexpr int kCols = SWIGLU ? kBlockM / 2 : kBlockM;  // output columns per CTA and tile
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  Control* ctl = reinterpret_cast<Control*>(ring + g.ring_bytes);
  // (kToPeers only) behind the control block; the tables come last.
  using Peers = PeerStage<kWide ? kMaxTokens : kMmaTokens>;
  Peers* peer_stage = reinterpret_cast<Peers*>(ctl + 1);
  uint32_t* tile_start = kToPeers ? reinterpret_cast<uint32_t*>(peer_stage + 1)
                                  : reinterpret_cast<uint32_t*>(ctl + 1);  // [E + 1]
  uint32_t* rows_of = tile_start + g.num_experts + 1;                      // [E] valid rows
  uint32_t* x_row0 = rows_of + g.num_experts;  // [E] first row in the token plane
  // kFromStaging: [E][world] rows that each source sends to the expert, or null when the table
  // does not fit (then the posted histograms are read again for every tile).
  uint32_t* src_rows = (kFromStaging && g.src_table != 0) ? x_row0 + g.num_experts : nullptr;
  const A2AParams& p = g.a2a;
  int parity = 0;

  const uint32_t cta_rank = kPair ? tc::cluster_ctarank() : 0u;
  const bool leader = cta_rank == 0u;
  const uint32_t worker = blockIdx.x / kCtas;   // tile-loop index
  const uint32_t workers = gridDim.x / kCtas;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile uint32_t* abort_flag = &ctl->abort_flag;
  const int w_blocks = ceil_div<int>(g.n_out, kCols * kCtas);
  const int num_kb = ceil_div<int>(g.k, kBlockK);

  // ---- set-up ---------------------------------------------------------------
  if (tid == 0) {
    ctl->abort_flag = 0;
    ctl->max_rows = 0;
    ctl->max_width = kUnit;
    ctl->best_limit = ~0ull;
    for (int s = 0; s < kMaxStages; ++s) {
      tc::mbar_init(&ctl->full[s], 1);
      tc::mbar_init(&ctl->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(&ctl->tmem_full[b], 1);
      tc::mbar_init(&ctl->tmem_empty[b], 8 * kCtas);  // epilogue warps of the tile
    }
    tc::fence_mbar_init();
    tc::tma_prefetch_desc(&tmap_w);
    tc::tma_prefetch_desc(&tmap_x.x64);
    tc::tma_prefetch_desc(&tmap_x.x16);
  }
  if (warp == 2) {
    if constexpr (kPair) {
      tc::tmem_alloc_2cta(&ctl->tmem_base, kTmemCols);
      tc::tmem_relinquish_2cta();
    } else {
      tc::tmem_alloc(&ctl->tmem_base, kTmemCols);
      tc::tmem_relinquish();
    }
  }
  ptx::wait_for_previous_kernels();
  if constexpr (!kFromStaging) ptx::let_next_kernel_start();
  if constexpr (kFromStaging || kToPeers) parity = static_cast<int>(ptx::ld_volatile(p.iter) & 1u);
  if constexpr (kFromStaging) {
    // Role of the dispatch receive phase: learn how many rows every source sends
    // to every local expert, lay the rows out, publish the per-expert totals.
    for (int le = tid; le < g.num_experts; le += blockDim.x) rows_of[le] = 0;
    __syncthreads();
    const WaitCtx w{p.status, p.timeout_ns, static_cast<uint32_t>(p.rank)};
    const uint32_t* all = reinterpret_cast<const uint32_t*>(p.peer[p.rank] + p.off_counts_all) +
                          static_cast<size_t>(parity) * p.world * p.num_experts;
    for (int idx = tid; idx < p.world * p.nle; idx += blockDim.x) {
      const int src = idx / p.nle;
      const int le = idx - src * p.nle;
      uint32_t v = 0;
      const bool ok = wait_until(all + static_cast<size_t>(src) * p.num_experts + p.rank * p.nle + le,
                                 PredNonZero{}, v, w, kPhaseDispatchCounts, src, 1u);
      if (!ok) ctl->abort_flag = 1;
      if (ok && v > 1u) atomicAdd(&rows_of[le], v - 1u);
      if (src_rows != nullptr) src_rows[le * p.world + src] = (ok && v > 1u) ? v - 1u : 0u;
    }
    __syncthreads();
    for (int le = tid; le < g.num_experts; le += blockDim.x) x_row0[le] = rows_of[le];
    __syncthreads();
    if (warp == 0) warp_exclusive_scan_smem(x_row0, g.num_experts, lane, false);
    __syncthreads();
    if (blockIdx.x == 0) {
      for (int le = tid; le < g.num_experts; le += blockDim.x) {
        if (g.out_num_tokens != nullptr) g.out_num_tokens[le] = static_cast<int32_t>(rows_of[le]);
        p.recv_count[le] = min(rows_of[le], static_cast<uint32_t>(p.cap));
      }
    }
  } else {
    __syncthreads();
  }
  for (int e = tid; e < g.num_experts; e += blockDim.x) {
    int rows;
    if constexpr (kFromStaging) {
      rows = static_cast<int>(min(rows_of[e], static_cast<uint32_t>(p.cap)));
    } else {
      rows = min(max(g.counts[e], 0), g.rows_per_expert);
      x_row0[e] = 0;
    }
    rows_of[e] = static_cast<uint32_t>(rows);
    if (rows > 0) atomicMax(&ctl->max_rows, static_cast<uint32_t>(rows));
  }
  if constexpr (kToPeers) {
    if (blockIdx.x == 0) {
      // Role of the combine send phase's first block: the dispatch that produced
      // these rows is over on this rank, so clear its flag set and move on.
      uint32_t* counts = reinterpret_cast<uint32_t*>(p.peer[p.rank] + p.off_counts) +
                         a2a_counts_index(p, parity, 0, 0);
      uint32_t* arrived =
          reinterpret_cast<uint32_t*>(p.peer[p.rank] + p.off_arrived) + parity * p.world;
      for (int q = tid; q < p.world * p.nle; q += blockDim.x) counts[q] = 0;
      if (tid < p.world) arrived[tid] = 0;
      reset_packed_flags(p, parity);
      __syncthreads();
      if (tid == 0) *p.iter = *p.iter + 1u;
    }
  }
  __syncthreads();

  // The most token rows a tile may have.  One tile per expert up to 256 rows: there an expert is
  // bound by its weights, which more tiles would only read again.  Above, the limit that
  // minimises (waves of tiles) x (time of a tile).  Per K block of 64 a tile of w rows takes 2 * w
  // cycles of MMAs, or as long as L2 needs for 16 KB of weights and 64 * w bytes of tokens per CTA
  // at 64 bytes per cycle; more than 256 rows leave no second accumulator, so their epilogue is
  // not hidden.  Every CTA computes the same.
  constexpr uint32_t kDrain = SWIGLU ? kDrainSwiglu : kDrainPlain;
  int limit = min(g.max_tokens, kWide ? kMaxTokens : kMmaTokens) / kUnit * kUnit;
  if (ctl->max_rows > static_cast<uint32_t>(min(limit, kMmaTokens))) {
    for (int cand = limit - kUnit * warp; 4 * cand >= limit; cand -= kUnit * (kThreads / 32)) {
      uint32_t tiles = 0, width = 0;
      for (int e = lane; e < g.num_experts; e += 32) {
        const Cut<kUnit> cut(static_cast<int>(rows_of[e]), cand);
        tiles += cut.tiles;
        width += cut.units * kUnit;
      }
      tiles = __reduce_add_sync(0xffffffffu, tiles);
      width = __reduce_add_sync(0xffffffffu, width);
      if (lane == 0) {
        const uint64_t waves = ceil_div<uint64_t>(static_cast<uint64_t>(tiles) * w_blocks, workers);
        const uint32_t w = width / tiles;
        const uint64_t cost = waves * (static_cast<uint64_t>(num_kb) * max(2u * w, 256u + w) +
                                       (cand > kMmaTokens ? kDrain * w : 0u));
        atomicMin(&ctl->best_limit, (cost << 16) | static_cast<uint64_t>(kMaxTokens - cand));
      }
    }
    __syncthreads();
    limit = kMaxTokens - static_cast<int>(ctl->best_limit & 0xffffu);
  }
  for (int e = tid; e < g.num_experts; e += blockDim.x) {
    const Cut<kUnit> cut(static_cast<int>(rows_of[e]), limit);
    tile_start[e] = static_cast<uint32_t>(cut.tiles * w_blocks);
    if (cut.tiles > 0) atomicMax(&ctl->max_width, static_cast<uint32_t>(cut.widest()));
  }
  __syncthreads();
  if (warp == 0) warp_exclusive_scan_smem(tile_start, g.num_experts, lane, true);
  tc::tc_fence_before_sync();
  __syncthreads();
  // The peer must see initialised barriers before anything arrives on them remotely.
  if constexpr (kPair) tc::cluster_sync();
  tc::tc_fence_after_sync();
  const uint32_t tmem_base = ctl->tmem_base;
  const uint32_t total_tiles = tile_start[g.num_experts];
  // As many stages as the launch's widest token tile leaves room for.
  const uint32_t stage_bytes = kWBytes + ctl->max_width / kCtas * kRowBytes;
  const uint32_t stages = min(g.ring_bytes / stage_bytes, static_cast<uint32_t>(kMaxStages));
  const bool two = !kWide || ctl->max_width <= kMmaTokens;  // two accumulators

  // ---- roles ----------------------------------------------------------------
  if (warp == 0) {
    if (tc::elect_one()) {
      uint32_t stage = 0, phase = 0;
      uint32_t pending = 0;        // stages that have been filled at least once
      uint32_t pending_phase = 0;  // parity of the phase each stage was last filled in
      bool ok = *abort_flag == 0u;
      int last_expert = -1;  // expert that `landed` refers to
      uint32_t landed = 0;   // bit s: the rows of source s for that expert have landed
      for (uint32_t t = worker; t < total_tiles && ok; t += workers) {
        const Tile c = locate<kUnit>(tile_start, rows_of, g.num_experts, limit, t);
        if constexpr (kFromStaging) {
          if (c.expert != last_expert) {
            last_expert = c.expert;
            landed = 0;
          }
          ok = wait_tile_sources(p, c.expert, c.first, min(c.first + c.width, c.rows), parity,
                                 src_rows, landed);
          if (!ok) {
            *abort_flag = 1u;
            break;
          }
        }
        // This CTA's share of the tokens of each MMA.
        const int n0 = kWide ? first_mma(c.width) : c.width;
        const int own0 = n0 / kCtas, own1 = (c.width - n0) / kCtas;
        const int row0 = static_cast<int>(x_row0[c.expert]) + c.first + static_cast<int>(cta_rank) * own0;
        const int row1 = row0 - static_cast<int>(cta_rank) * own0 + n0 + static_cast<int>(cta_rank) * own1;
        const int x_plane = kFromStaging ? 0 : c.expert;
        const int w_row = (c.w_blk * kCtas + static_cast<int>(cta_rank)) * kCols;
        const uint32_t tx = kCtas * kWBytes + static_cast<uint32_t>(c.width) * kRowBytes;
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = tc::mbar_wait(&ctl->empty[stage], phase ^ 1u, abort_flag, kWaitLimitNs);
          if (!ok) break;
          uint8_t* w_dst = ring + stage * stage_bytes;
          uint8_t* x_dst = w_dst + kWBytes;
          uint64_t* full = &ctl->full[stage];
          pending |= 1u << stage;
          pending_phase = (pending_phase & ~(1u << stage)) | (phase << stage);
          // The bytes of both CTAs are counted on the leader's barrier, which only the leader
          // arms.
          if (leader) tc::mbar_arrive_expect_tx(full, tx);
          if constexpr (SWIGLU) {
            if constexpr (kPair)
              tc::tma_load_5d_2cta(w_dst, &tmap_w, full, kb * kBlockK, 0, 0, w_row / 8, c.expert);
            else
              tc::tma_load_5d(w_dst, &tmap_w, full, kb * kBlockK, 0, 0, w_row / 8, c.expert);
          } else {
            load_rows<kPair>(w_dst, &tmap_w, full, kb * kBlockK, w_row, c.expert);
          }
          int r = 0;
          for (; r + 64 <= own0; r += 64, x_dst += 64 * kRowBytes)
            load_rows<kPair>(x_dst, &tmap_x.x64, full, kb * kBlockK, row0 + r, x_plane);
          for (; r < own0; r += 16, x_dst += 16 * kRowBytes)
            load_rows<kPair>(x_dst, &tmap_x.x16, full, kb * kBlockK, row0 + r, x_plane);
          if constexpr (kWide) {
            r = 0;
            for (; r + 64 <= own1; r += 64, x_dst += 64 * kRowBytes)
              load_rows<kPair>(x_dst, &tmap_x.x64, full, kb * kBlockK, row1 + r, x_plane);
            for (; r < own1; r += 16, x_dst += 16 * kRowBytes)
              load_rows<kPair>(x_dst, &tmap_x.x16, full, kb * kBlockK, row1 + r, x_plane);
          }
          if (++stage == stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      // (Nothing is waited for any more that another stream or rank has to do.)
      if constexpr (kFromStaging) ptx::let_next_kernel_start();
      if (!ok || *abort_flag != 0u) {
        // Give the loads already issued a bounded time to land before the CTA
        // leaves: their destination is this CTA's shared memory.
        const uint64_t t0 = ptx::globaltimer_ns();
        for (uint32_t s = 0; s < stages; ++s) {
          if (!((pending >> s) & 1u)) continue;
          // (The non-leader of a pair has no barrier of its own to watch; it just sits
          // out the time limit, which is far longer than any load takes.)
          while (!leader || !tc::mbar_try_wait(&ctl->full[s], (pending_phase >> s) & 1u)) {
            if (ptx::globaltimer_ns() - t0 > 100000000ull) break;  // 100 ms in total
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (leader && tc::elect_one()) {
      uint32_t stage = 0, phase = 0, local = 0;
      bool ok = *abort_flag == 0u;
      for (uint32_t t = worker; t < total_tiles && ok; t += workers, ++local) {
        const Tile c = locate<kUnit>(tile_start, rows_of, g.num_experts, limit, t);
        const int n0 = kWide ? first_mma(c.width) : c.width, n1 = c.width - n0;
        const uint32_t idesc = tc::make_instr_desc(1u, kBlockM * kCtas, n0);
        const uint32_t idesc1 = tc::make_instr_desc(1u, kBlockM * kCtas, n1);
        const uint32_t buf = two ? local & 1u : 0u;
        const uint32_t use = two ? local >> 1 : local;  // how often this accumulator was used before
        ok = tc::mbar_wait(&ctl->tmem_empty[buf], (use & 1u) ^ 1u, abort_flag, kWaitLimitNs);
        if (!ok) break;
        tc::tc_fence_after_sync();
        const uint32_t tmem_d = tmem_base + buf * kMmaTokens;
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = tc::mbar_wait(&ctl->full[stage], phase, abort_flag, kWaitLimitNs);
          if (!ok) break;
          tc::tc_fence_after_sync();
          const uint8_t* w_src = ring + stage * stage_bytes;
          const uint64_t w_desc = tc::make_smem_desc_sw128(w_src);
          const uint64_t x_desc = tc::make_smem_desc_sw128(w_src + kWBytes);
#pragma unroll
          for (int k = 0; k < kBlockK / kUmmaK; ++k) {
            const uint64_t wd = tc::advance_smem_desc(w_desc, k * kUmmaK * 2);
            const uint64_t xd = tc::advance_smem_desc(x_desc, k * kUmmaK * 2);
            if constexpr (kPair) tc::mma_f16_ss_2cta(tmem_d, wd, xd, idesc, (kb | k) != 0);
            else tc::mma_f16_ss(tmem_d, wd, xd, idesc, (kb | k) != 0);
          }
          if constexpr (kWide) {
            if (n1 > 0) {
              const uint64_t x1_desc = tc::advance_smem_desc(x_desc, n0 / kCtas * kRowBytes);
#pragma unroll
              for (int k = 0; k < kBlockK / kUmmaK; ++k)
                tc::mma_f16_ss_2cta(tmem_d + n0, tc::advance_smem_desc(w_desc, k * kUmmaK * 2),
                                    tc::advance_smem_desc(x1_desc, k * kUmmaK * 2), idesc1,
                                    (kb | k) != 0);
            }
          }
          // Stage reusable (in both CTAs of a pair) once these MMAs have read it.
          if constexpr (kPair) tc::mma_commit_2cta(&ctl->empty[stage], 0x3);
          else tc::mma_commit(&ctl->empty[stage]);
          if (++stage == stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (ok) {
          if constexpr (kPair) tc::mma_commit_2cta(&ctl->tmem_full[buf], 0x3);
          else tc::mma_commit(&ctl->tmem_full[buf]);
        }
      }
    }
    __syncwarp();
  } else if (warp >= 4) {
    const int ew = (warp - 4) & 3;   // tensor-memory lanes [32 * ew, +32)
    const int wg = (warp - 4) >> 2;  // 16-token groups wg, wg + 2, wg + 4, ...
    const int n_tid = tid - 128;     // 0..255 over the eight warps
    const int lt = n_tid & 127;      // thread of the warp group
    const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(ew * 32) << 16);
    uint32_t local = 0;
    uint32_t pending_signals = 0;  // kToPeers, warp 4: queued arrival adds
    bool ok = *abort_flag == 0u;
    for (uint32_t t = worker; t < total_tiles && ok; t += workers, ++local) {
      const Tile c = locate<kUnit>(tile_start, rows_of, g.num_experts, limit, t);
      const uint32_t buf = two ? local & 1u : 0u;
      ok = tc::mbar_wait(&ctl->tmem_full[buf], (two ? local >> 1 : local) & 1u, abort_flag, kWaitLimitNs);
      // All eight warps leave together or not at all: the barriers below must never be
      // entered by only some of them.
      {
        uint32_t all_ok;
        asm volatile(
            "{\n\t"
            ".reg .pred p, q;\n\t"
            "setp.ne.u32 q, %1, 0;\n\t"
            "bar.red.and.pred p, 1, 256, q;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t"
            "}\n"
            : "=r"(all_ok)
            : "r"(ok ? 1u : 0u)
            : "memory");
        ok = all_ok != 0u;
      }
      if (!ok) break;
      tc::tc_fence_after_sync();
      const int groups = c.width >> 4;
      const int live = min(c.width, c.rows - c.first);  // tokens of the tile that exist
      const int col0 = (c.w_blk * kCtas + static_cast<int>(cta_rank)) * kCols;
      if constexpr (kFromStaging) {
        // The first block of columns also records where the rows came from.
        for (int n = n_tid; col0 == 0 && n < live; n += 256) {
          const int row = c.first + n;
          const uint8_t* slot = p.peer[p.rank] + p.off_disp_stage +
                                (static_cast<size_t>(x_row0[c.expert]) + row) * p.slot_bytes;
          const int4 tr = ptx::ld_cg_v4(slot + p.trailer_off);
          uint2 rs;
          rs.x = (static_cast<uint32_t>(tr.w) & 0xffffu) | (static_cast<uint32_t>(tr.y) << 16);
          rs.y = static_cast<uint32_t>(tr.x);
          p.row_src[static_cast<size_t>(c.expert) * p.cap + row] = rs;
        }
      }
      if constexpr (kToPeers) {
        // Where each token's row goes, and whose token it is.  (The barrier above comes after
        // the last use of the previous tile's table.)
        for (int n = n_tid; n < c.width; n += 256) {
          unsigned long long off = 0;
          uint32_t sig_token = kNoSignal, sig_group = 0;
          if (n < live) {
            const uint2 rs = p.row_src[static_cast<size_t>(c.expert) * p.cap + c.first + n];
            const int src_rank = static_cast<int>(rs.x & 0xffffu);
            const uint32_t k = rs.x >> 16;
            const uint32_t token = rs.y;
            if (token < static_cast<uint32_t>(p.max_tokens) && k < static_cast<uint32_t>(p.topk) &&
                src_rank < p.world) {
              sig_token = token;
              sig_group = static_cast<uint32_t>((src_rank / p.dp_size) * p.dp_size);
              off = p.off_comb_stage +
                    (static_cast<size_t>(token) * p.topk + k) * (static_cast<size_t>(g.n_out) * 2);
            } else if (p.debug_checks) {
              report_failure(p.status, kBadToken, kPhaseCombinePayload, src_rank, p.max_tokens,
                             token, p.rank);
            }
          }
          peer_stage->token[n] = sig_token;
          peer_stage->group[n] = sig_group;
          peer_stage->row_off[n] = off;
        }
        asm volatile("bar.sync 4, 256;" ::: "memory");
      }
      // A thread's values lie across token rows; each group of 16 tokens passes through shared
      // memory so that rows leave in 16-byte pieces.  The wide form, whose accumulator may be the
      // only one, hands it back when its last group is in registers; the other, which has two, after
      // the tile (earlier was slower there).
      const uint32_t t_acc = t_lane + buf * kMmaTokens;
      auto hand_back = [&] {
        tc::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          if constexpr (kPair) tc::mbar_arrive_on_leader(&ctl->tmem_empty[buf]);
          else tc::mbar_arrive(&ctl->tmem_empty[buf]);
        }
      };
      if (kWide && wg >= groups) hand_back();
#pragma unroll 1
      for (int grp = wg, alt = 0; grp < groups; grp += 2, alt ^= 1) {
        uint32_t lo[8], hi[8];
        load_group(t_acc + grp * 16, lo, hi);
        tc::tmem_ld_wait();
        if (kWide && grp + 2 >= groups) hand_back();
        uint8_t(*seg)[kSegBytes] = ctl->seg[wg][alt];
        if constexpr (SWIGLU) {
          // Lanes 0-7 of every 16 are gate rows, 8-15 the up rows of the same columns.
          stmatrix_x4_trans(&seg[8 * (lane >> 4) + (lane & 7)][(ew * 16 + ((lane >> 3) & 1) * 8) * 2],
                            swiglu_pair(lo[0], lo[1], lo[2], lo[3]),
                            swiglu_pair(hi[0], hi[1], hi[2], hi[3]),
                            swiglu_pair(lo[4], lo[5], lo[6], lo[7]),
                            swiglu_pair(hi[4], hi[5], hi[6], hi[7]));
        } else {
#pragma unroll
          for (int b = 0; b < 2; ++b)
            stmatrix_x4_trans(&seg[8 * b + (lane & 7)][(ew * 32 + (lane >> 3) * 8) * 2],
                              pack_bits(lo[4 * b], lo[4 * b + 1]),
                              pack_bits(lo[4 * b + 2], lo[4 * b + 3]),
                              pack_bits(hi[4 * b], hi[4 * b + 1]),
                              pack_bits(hi[4 * b + 2], hi[4 * b + 3]));
        }
        sync_group(wg);
        constexpr int kPieces = kCols / 8;  // 16-byte pieces of a token's row segment
        const int piece = lt % kPieces;
        const int col = col0 + piece * 8;
#pragma unroll
        for (int tok16 = lt / kPieces; tok16 < 16; tok16 += 128 / kPieces) {
          const int n = grp * 16 + tok16;
          const int4 v = *reinterpret_cast<const int4*>(&seg[tok16][piece * 16]);
          if (col + 8 > g.n_out) continue;
          if constexpr (kToPeers) {
            if (peer_stage->token[n] != kNoSignal) {
              const uint32_t first_rank = peer_stage->group[n];
              const size_t off = peer_stage->row_off[n] + static_cast<size_t>(col) * 2;
              for (int r = 0; r < min(p.dp_size, 8); ++r) ptx::st_v4(p.peer[first_rank + r] + off, v);
            }
          } else if (n < live) {
            *reinterpret_cast<int4*>(g.out + c.expert * g.out_stride_e +
                                     static_cast<int64_t>(c.first + n) * g.out_stride_row + col) = v;
          }
        }
      }
      if constexpr (!kWide) hand_back();
      if constexpr (kToPeers) {
        // Arrival is counted in columns: this tile's share of each row.  The adds are queued
        // and flushed behind ONE system-scope fence for as many tiles as the queue holds.
        asm volatile("bar.sync 4, 256;" ::: "memory");
        if (warp == 4 && col0 < g.n_out) {
          const uint32_t units = static_cast<uint32_t>(min(kCols, g.n_out - col0));
          if (pending_signals + c.width > kQueue) {
            flush(p, peer_stage, pending_signals, lane);
            pending_signals = 0;
          }
          for (int j0 = 0; j0 < c.width; j0 += 32) {
            const uint32_t token = j0 + lane < c.width ? peer_stage->token[j0 + lane] : kNoSignal;
            const bool there = token != kNoSignal;
            const uint32_t mask = __ballot_sync(0xffffffffu, there);
            if (there) {
              const uint32_t at = pending_signals + __popc(mask & ((1u << lane) - 1u));
              peer_stage->q_token[at] = token;
              peer_stage->q_group_units[at] = peer_stage->group[j0 + lane] | (units << 8);
            }
            pending_signals += __popc(mask);
          }
          __syncwarp();
        }
      }
    }
    if constexpr (kToPeers) {
      // What is still queued (also after a failed wait: rows that were stored are announced).
      if (warp == 4 && pending_signals > 0) flush(p, peer_stage, pending_signals, lane);
    }
  }

  // ---- teardown -------------------------------------------------------------
  tc::tc_fence_before_sync();
  __syncthreads();
  // Neither CTA of a pair may leave while the other can still touch its shared or
  // tensor memory.
  if constexpr (kPair) tc::cluster_sync();
  if (warp == 2) {
    tc::tc_fence_after_sync();
    if constexpr (kPair) tc::tmem_dealloc_2cta(tmem_base, kTmemCols);
    else tc::tmem_dealloc(tmem_base, kTmemCols);
  }
  if (tid == 0 && ctl->abort_flag != 0u && g.status != nullptr) *g.status = 1u;
  (void)parity;
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                   const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    CUDA_CHECK(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
    PPLX_CHECK(q == cudaDriverEntryPointSuccess && p != nullptr,
               "cuTensorMapEncodeTiled is not available in this driver");
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

CUtensorMap encode_map(int rank, const void* base, const cuuint64_t* dims, const cuuint64_t* strides,
                       const cuuint32_t* box) {
  PPLX_CHECK(reinterpret_cast<uintptr_t>(base) % 16 == 0, "operand base must be 16-byte aligned");
  const cuuint32_t elem_strides[5] = {1, 1, 1, 1, 1};
  CUtensorMap map;
  const CUresult r = encode_tiled()(
      &map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(base), dims, strides, box,
      elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  PPLX_CHECK(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed with code " << static_cast<int>(r));
  return map;
}

void check_strides(int64_t stride_row_elems, int64_t stride_expert_elems) {
  PPLX_CHECK((stride_row_elems * 2) % 16 == 0 && (stride_expert_elems * 2) % 16 == 0,
             "operand strides must be multiples of 16 bytes (8 bf16 elements)");
}

// [planes, rows, k] bf16 with k contiguous; tiles of 64 x box_rows x 1, 128-byte swizzle,
// out-of-range elements read as zero.
CUtensorMap make_operand_map(const void* base, int64_t planes, int64_t rows, int64_t k,
                             int64_t stride_row_elems, int64_t stride_plane_elems, int box_rows) {
  check_strides(stride_row_elems, stride_plane_elems);
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(k), static_cast<cuuint64_t>(rows),
                              static_cast<cuuint64_t>(planes)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(stride_row_elems) * 2,
                                 static_cast<cuuint64_t>(stride_plane_elems) * 2};
  const cuuint32_t box[3] = {kBlockK, static_cast<cuuint32_t>(box_rows), 1};
  return encode_map(3, base, dims, strides, box);
}

// 128 weight rows per tile.  Plain: consecutive ones.  SwiGLU: [experts][2 * n_out][k] seen as
// [experts][n_out / 8][gate, up][8][k], so that a box of 8 x 2 x 8 rows is eight gate rows, the
// eight up rows of the same columns, the next eight gate rows, ...
CUtensorMap make_weight_map(const GroupedGemmCall& c) {
  if (!c.swiglu)
    return make_operand_map(c.w, c.num_experts, c.n_out, c.k, c.w_stride_row, c.w_stride_e, kBlockM);
  check_strides(c.w_stride_row, c.w_stride_e);
  const cuuint64_t row = static_cast<cuuint64_t>(c.w_stride_row) * 2;
  const cuuint64_t dims[5] = {static_cast<cuuint64_t>(c.k), 8, 2,
                              static_cast<cuuint64_t>(c.n_out / 8),
                              static_cast<cuuint64_t>(c.num_experts)};
  const cuuint64_t strides[4] = {row, row * static_cast<cuuint64_t>(c.n_out), row * 8,
                                 static_cast<cuuint64_t>(c.w_stride_e) * 2};
  const cuuint32_t box[5] = {kBlockK, 8, 2, 8, 1};
  return encode_map(5, c.w, dims, strides, box);
}

TokenMaps make_token_maps(const void* base, int64_t planes, int64_t rows, int64_t k,
                          int64_t stride_row, int64_t stride_plane) {
  return {make_operand_map(base, planes, rows, k, stride_row, stride_plane, 64),
          make_operand_map(base, planes, rows, k, stride_row, stride_plane, 16)};
}

// The per-source table is kept in shared memory when it is at most this many entries.
constexpr size_t kMaxSrcEntries = 2048;

template <bool SWIGLU, bool kFromStaging, bool kToPeers, bool kPair, bool kWide>
void launch_one(const CUtensorMap& tmap_w, const TokenMaps& tmap_x, GroupedGemmArgs g, int grid,
                cudaStream_t stream) {
  auto* kernel = grouped_gemm_kernel<SWIGLU, kFromStaging, kToPeers, kPair, kWide>;
  const size_t src_entries =
      (kFromStaging && g.src_table != 0) ? static_cast<size_t>(g.num_experts) * g.a2a.world : 0;
  const size_t fixed = 1024 + sizeof(Control) + (kToPeers ? sizeof(PeerStage<kWide ? kMaxTokens : kMmaTokens>) : 0) +
                       sizeof(uint32_t) * (3 * static_cast<size_t>(g.num_experts) + 1 + src_entries);
  // The stages take what the tables leave; kMaxExperts and kMaxSrcEntries leave room for at
  // least three of the widest tiles (four beside the tables of 256 experts).
  constexpr size_t kSmem = 227 * 1024;
  static_assert(kSmem - (1024 + sizeof(Control) + sizeof(PeerStage<kMaxTokens>) +
                         sizeof(uint32_t) * (3 * kMaxExperts + 1 + kMaxSrcEntries)) >=
                    3 * (kWBytes + kMaxTokens / 2 * kRowBytes) + 1024,
                "too little shared memory for the stages");
  g.ring_bytes = static_cast<uint32_t>((kSmem - fixed) & ~static_cast<size_t>(1023));
  const size_t smem = fixed + g.ring_bytes;
  CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(smem)));
  void* params[] = {const_cast<CUtensorMap*>(&tmap_w), const_cast<TokenMaps*>(&tmap_x), &g};
  CUDA_CHECK(launch_after_previous(reinterpret_cast<const void*>(kernel),
                                   dim3(kPair ? (grid & ~1) : grid), dim3(kThreads), params, smem,
                                   stream, kPair ? 2 : 1));
}

// Tiles of up to 512 token rows, from an expected mean of 224 rows per expert on: from about there
// an expert may have more than 256 (and every form takes any number of rows).  8 experts, up /
// down projection of Mixtral 8x7B, tiles of at most 256 and at most 512 rows: 300 rows each 547 /
// 276 and 498 / 229 us, 512 rows 750 / 550 and 770 / 383 us, 1024 rows 1370 / 800 and 1410 / 685 us.
// With few rows, where the weights bound the kernel, it costs 1 to 2 us: 128 rows 325.5 / 169.8
// and 327.7 / 171.0 us.
bool want_wide(const GroupedGemmCall& c) {
  const int64_t rows = c.expected_total_rows > 0
                           ? c.expected_total_rows
                           : static_cast<int64_t>(c.num_experts) * c.rows_per_expert;
  return c.half_n == 0 && rows >= 224 * static_cast<int64_t>(c.num_experts);
}

template <bool SWIGLU, bool kFromStaging, bool kToPeers>
void launch_variant(const CUtensorMap& tmap_w, const TokenMaps& tmap_x, const GroupedGemmArgs& g,
                    const GroupedGemmCall& c, cudaStream_t stream) {
  const int grid = c.num_sms > 0 ? c.num_sms : get_sm_count();
  if (c.cta_pair == 0 || grid < 2)
    launch_one<SWIGLU, kFromStaging, kToPeers, false, false>(tmap_w, tmap_x, g, grid, stream);
  else if (want_wide(c))
    launch_one<SWIGLU, kFromStaging, kToPeers, true, true>(tmap_w, tmap_x, g, grid, stream);
  else
    launch_one<SWIGLU, kFromStaging, kToPeers, true, false>(tmap_w, tmap_x, g, grid, stream);
}

void check_common(const GroupedGemmCall& c) {
  PPLX_CHECK(c.num_experts > 0 && c.num_experts <= kMaxExperts, "num_experts out of range");
  PPLX_CHECK(c.k > 0 && c.k % 8 == 0, "K must be a positive multiple of 8");
  PPLX_CHECK(c.n_out > 0 && c.n_out % 8 == 0, "the output width must be a positive multiple of 8");
  PPLX_CHECK(c.half_n == 0 || (c.half_n % 8 == 0 && c.half_n >= 16 && c.half_n <= 128),
             "half_n must be a multiple of 8 in [16, 128]");
}

GroupedGemmArgs base_args(const GroupedGemmCall& c) {
  GroupedGemmArgs g{};
  g.counts = c.counts;
  g.out = static_cast<__nv_bfloat16*>(c.out);
  g.out_stride_e = c.out_stride_e;
  g.out_stride_row = c.out_stride_row;
  g.status = c.status;
  g.num_experts = c.num_experts;
  g.rows_per_expert = c.rows_per_expert;
  g.n_out = c.n_out;
  g.k = c.k;
  g.max_tokens = c.half_n > 0 ? 2 * c.half_n : kMaxTokens;
  return g;
}

}  // namespace

void launch_grouped_gemm(const GroupedGemmCall& c, cudaStream_t stream) {
  check_common(c);
  PPLX_CHECK(reinterpret_cast<uintptr_t>(c.out) % 16 == 0 && c.out_stride_row % 8 == 0 &&
                 c.out_stride_e % 8 == 0,
             "the output must be 16-byte aligned");
  const TokenMaps tmap_x = make_token_maps(c.x, c.num_experts, c.rows_per_expert, c.k,
                                              c.x_stride_row, c.x_stride_e);
  GroupedGemmArgs g = base_args(c);
  const CUtensorMap tmap_w = make_weight_map(c);
  if (c.swiglu) launch_variant<true, false, false>(tmap_w, tmap_x, g, c, stream);
  else launch_variant<false, false, false>(tmap_w, tmap_x, g, c, stream);
}

void launch_gemm_from_staging(const GroupedGemmCall& c, const A2AParams& p,
                              int32_t* out_num_tokens, cudaStream_t stream) {
  check_common(c);
  PPLX_CHECK(c.swiglu, "the staging-fed GEMM is the SwiGLU up projection");
  PPLX_CHECK(p.scale_bytes == 0 && p.hidden_bytes == p.hidden_dim * 2,
             "the staging-fed GEMM needs a bf16 dispatch payload without scales");
  PPLX_CHECK(c.k == p.hidden_dim && c.num_experts == p.nle && c.rows_per_expert >= p.cap,
             "shape mismatch between the GEMM and the all-to-all");
  PPLX_CHECK(reinterpret_cast<uintptr_t>(c.out) % 16 == 0 && c.out_stride_row % 8 == 0 &&
                 c.out_stride_e % 8 == 0,
             "the output must be 16-byte aligned");
  // Tokens: [1][world * region_slots][hidden] bf16 view of this rank's packed staging.
  const int64_t slots = static_cast<int64_t>(p.world) * p.region_slots;
  const TokenMaps tmap_x = make_token_maps(p.peer[p.rank] + p.off_disp_stage, 1, slots,
                                              p.hidden_dim, p.slot_bytes / 2,
                                              slots * p.slot_bytes / 2);
  GroupedGemmArgs g = base_args(c);
  const CUtensorMap tmap_w = make_weight_map(c);
  g.out_num_tokens = out_num_tokens;
  g.a2a = p;
  g.src_table = static_cast<size_t>(p.nle) * p.world <= kMaxSrcEntries ? 1 : 0;
  launch_variant<true, true, false>(tmap_w, tmap_x, g, c, stream);
}

void launch_gemm_to_peers(const GroupedGemmCall& c, const A2AParams& p, cudaStream_t stream) {
  check_common(c);
  PPLX_CHECK(!c.swiglu, "the peer-storing GEMM is the plain down projection");
  PPLX_CHECK(c.n_out == p.hidden_dim && c.num_experts == p.nle && c.rows_per_expert >= p.cap,
             "shape mismatch between the GEMM and the all-to-all");
  PPLX_CHECK(c.counts == reinterpret_cast<const int32_t*>(p.recv_count),
             "counts must be the all-to-all's received-row counts");
  PPLX_CHECK(p.dp_size <= 8, "at most 8 replicas per DP group");
  const TokenMaps tmap_x = make_token_maps(c.x, c.num_experts, c.rows_per_expert, c.k,
                                              c.x_stride_row, c.x_stride_e);
  GroupedGemmArgs g = base_args(c);
  const CUtensorMap tmap_w = make_weight_map(c);
  g.out = nullptr;
  g.a2a = p;
  launch_variant<false, false, true>(tmap_w, tmap_x, g, c, stream);
}

}  // namespace pplx
