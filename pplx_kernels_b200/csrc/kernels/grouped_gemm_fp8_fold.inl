// fp8 expert GEMM with fp32 scales (included by grouped_gemm_fp8_sm100.cu).
//
// The WEIGHTS are the M operand of the MMAs and the tokens the N operand: a tile is kHalves
// blocks of 128 weight rows (SwiGLU: 128 gate and 128 up rows, which is one scale block of the
// result; plain: 128 output columns) times a token tile of 16 to kMaxTokens rows of the expert,
// in steps of 16.  Expert parallelism leaves an expert with anything from one row to a few
// thousand.  With the tokens as M (the first form of this kernel) every expert was padded to 128
// rows: at 61 tokens over 128 experts the tensor and CUDA cores worked on 32 times the rows that
// exist, and what should have been a stream of weights at DRAM rate (62 us) took 146 us.  With
// the tokens as N the work per weight byte follows the rows there are, so few rows leave the
// kernel bound by the weight stream, and a large expert is cut into equal tiles instead of full
// ones and a nearly empty last one.
//
// fp32 scales per 128 columns of K are not the hardware's block-scale format, so each 128-wide
// K block is multiplied into one of four scratch accumulators in tensor memory and folded, times
// the two scales, into running sums in REGISTERS by eight warps.  Tensor memory is read in the
// 16x256b shape, so that a thread holds four weight rows of every fourth pair of tokens instead
// of one row of all tokens: the products (token scale) * (weight scale), which a warp of their
// own puts into shared memory, are then one shared-memory word per four FMAs (per FMA, as the
// row shape would need, the reads alone took longer than the MMAs), and the folding is a packed
// two-wide FMA.  Each warp group of four folds every second group of 16 tokens.
//
// The token tile is limited so that a thread's sums stay in its registers (a few spilled words
// made the K loop half as slow again: with this much shared memory there is no L1 to hold them),
// and the epilogue is kept short: with one or two tiles per CTA its instructions come from DRAM.
// An MMA of 128 x (16 to 64) takes about 90 cycles whatever its width (it is bound by reading the
// 128 weight rows from shared memory), so a K block of 256 weight rows takes 0.4 us: half of what
// its 32 KB need from DRAM with all SMs at it.
//
// Up projection, kernel times before and after: 125 of 128 experts of 768 x 2 x 2048 with 4 rows
// each 146 -> 71 us (5.5 TB/s), 32 experts of 2048 x 2 x 7168 with 32 rows 205 -> 152 us
// (6.2 TB/s); down 104 -> 85 us for the latter.
//
// Roles: warp 0 TMA producer, warp 1 MMA issuer, warp 2 tensor-memory allocation, warp 3
// scales, warps 4-11 fold and epilogue.
namespace pplx {
namespace {
namespace fold {

using namespace tok;

constexpr int kMaxStages = 12;
constexpr int kSegBytes = 256 + 16;  // 128 columns of bf16 of one token, padded
constexpr int kBuffers = 4;          // scratch accumulators of 128 columns of tensor memory

template <int kHalves>
struct Shape {
  static constexpr int kMaxTokens = 128 / kHalves;
  static constexpr int kGroups = kMaxTokens / 32;   // 16-token groups per folding thread
  static constexpr uint32_t kWBytes = kHalves * kBlockM * kBlockKBytes;
};

struct Tile {
  int expert;
  int w_blk;    // block of 128 output columns
  int first;    // first token row of the tile inside its expert
  int width;    // token rows of the tile, a multiple of 16
  int rows;     // valid rows of the expert
};

struct Control {
  uint64_t full[kMaxStages];
  uint64_t empty[kMaxStages];
  uint64_t part_full[kBuffers];   // scratch accumulator and scale products of a K block are there
  uint64_t part_empty[kBuffers];  // ... have been folded
  uint32_t tmem_base;
  uint32_t abort_flag;
  uint32_t max_tokens;            // widest token tile of this launch
  uint32_t pad;
  rows::Barriers row_bar;         // kMany
  alignas(16) float scales[kBuffers][128];  // [half * kMaxTokens + token]
  float amax[2][4][64];                     // SwiGLU: [warp group][warp][token of the group's]
  float inv_scale[2][64];
  alignas(16) uint8_t seg[2][2][16][kSegBytes];  // [warp group][alternating][token][column]
};
static_assert(sizeof(Control::seg) >= rows::kScratchBytes, "scratch of the form for many rows");

// Tiles of an expert are ordered with the token tile fastest: CTAs that run at the same time
// share a block of weights in L2.
template <int kHalves>
__device__ __forceinline__ Tile locate(const uint32_t* tile_start, const uint32_t* rows_of,
                                       int num_experts, uint32_t t) {
  Tile c;
  c.expert = find_group(tile_start, num_experts, t);
  c.rows = static_cast<int>(rows_of[c.expert]);
  const int tiles = token_tiles(c.rows, Shape<kHalves>::kMaxTokens);
  const uint32_t rem = t - tile_start[c.expert];
  c.w_blk = static_cast<int>(rem / tiles);
  c.width = token_width(c.rows, tiles);
  c.first = static_cast<int>(rem - static_cast<uint32_t>(c.w_blk) * tiles) * c.width;
  return c;
}

__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// A group of 16 tokens times this warp's 32 weight rows, as a thread holds it: pair[2 * q + b] is
// tokens {8 * b + 2 * (t % 4), + 1} of row 8 * q + t / 4.
struct Group {
  uint64_t pair[8];
};

// acc += part * scale; `scales` points at the group's 16 products.
__device__ __forceinline__ void fold_group(Group& acc, const uint32_t (&lo)[8],
                                           const uint32_t (&hi)[8], const float* scales, int lane) {
#pragma unroll
  for (int b = 0; b < 2; ++b) {
    const uint64_t s = *reinterpret_cast<const uint64_t*>(scales + 8 * b + 2 * (lane & 3));
    fma2(acc.pair[b], pack2(lo[4 * b], lo[4 * b + 1]), s);
    fma2(acc.pair[2 + b], pack2(lo[4 * b + 2], lo[4 * b + 3]), s);
    fma2(acc.pair[4 + b], pack2(hi[4 * b], hi[4 * b + 1]), s);
    fma2(acc.pair[6 + b], pack2(hi[4 * b + 2], hi[4 * b + 3]), s);
  }
}

__device__ __forceinline__ uint32_t bf16_pair(uint64_t v) {
  const float2 f = unpack2(v);
  const __nv_bfloat162 h = __floats2bfloat162_rn(f.x, f.y);
  return *reinterpret_cast<const uint32_t*>(&h);
}

struct FoldLoop {
  Control* ctl;
  volatile uint32_t* abort_flag;
  uint32_t t_lane;     // this warp's tensor-memory lanes
  int num_kb, wg, lane;
};

// The K loop of a folding warp that owns kOwn groups of the tile.  The number of groups is a
// template parameter so that the loop has no branches around its sums: with them, sums were moved
// between registers from group to group.  False: a wait ran out.
template <int kHalves, int kOwn>
__device__ __forceinline__ bool fold_k_loop(const FoldLoop& f,
                                            Group (&acc)[kHalves][Shape<kHalves>::kGroups],
                                            uint32_t& round) {
  using S = Shape<kHalves>;
  // Groups whose columns are in flight together: what the registers beside the sums hold.
  constexpr int kBatch = kOwn * kHalves <= 2 ? (kOwn > 0 ? kOwn : 1) : 2 / kHalves;
#pragma unroll
  for (int h = 0; h < kHalves; ++h) {
#pragma unroll
    for (int i = 0; i < kOwn; ++i) {
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[h][i].pair[j] = 0;
    }
  }
#pragma unroll 1
  for (int kb = 0; kb < f.num_kb; ++kb, ++round) {
    const uint32_t buf = round % kBuffers;
    if (!tc::mbar_wait(&f.ctl->part_full[buf], (round / kBuffers) & 1u, f.abort_flag,
                       kWaitLimitNs))
      return false;
    tc::tc_fence_after_sync();
    const uint32_t t_part = f.t_lane + buf * 128 + f.wg * 16;
    const float* scales = f.ctl->scales[buf] + f.wg * 16;
#pragma unroll
    for (int i0 = 0; i0 < kOwn; i0 += kBatch) {
      uint32_t lo[kBatch][kHalves][8], hi[kBatch][kHalves][8];
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        if (i0 + j >= kOwn) continue;
#pragma unroll
        for (int h = 0; h < kHalves; ++h)
          load_group(t_part + h * S::kMaxTokens + (i0 + j) * 32, lo[j][h], hi[j][h]);
      }
      tc::tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        if (i0 + j >= kOwn) continue;
#pragma unroll
        for (int h = 0; h < kHalves; ++h)
          fold_group(acc[h][i0 + j], lo[j][h], hi[j][h],
                     scales + h * S::kMaxTokens + (i0 + j) * 32, f.lane);
      }
    }
    tc::tc_fence_before_sync();
    __syncwarp();
    if (f.lane == 0) tc::mbar_arrive(&f.ctl->part_empty[buf]);
  }
  return true;
}

template <int kHalves, int kOwn = Shape<kHalves>::kGroups>
__device__ __forceinline__ bool fold_tile(const FoldLoop& f, int own,
                                          Group (&acc)[kHalves][Shape<kHalves>::kGroups],
                                          uint32_t& round) {
  if constexpr (kOwn > 0) {
    if (own < kOwn) return fold_tile<kHalves, kOwn - 1>(f, own, acc, round);
  }
  return fold_k_loop<kHalves, kOwn>(f, acc, round);
}

// kMany: the set-up, then the form for many rows per expert.  (A kernel of its own: with both forms in
// one, chosen by the row counts on the device, the registers of either were worse and every size was
// 5 to 10 % slower.)
template <bool kSwiGLUQuant, bool kFromStaging, bool kToPeers, bool kMany>
__global__ void __launch_bounds__(kThreads, 1)
    grouped_gemm_fp8_fold_kernel(const __grid_constant__ CUtensorMap tmap_w,
                                 const __grid_constant__ CUtensorMap tmap_x64,
                                 const __grid_constant__ CUtensorMap tmap_x16,
                                 const __grid_constant__ Fp8GemmArgs g) {
  static_assert(!(kFromStaging && kToPeers) && !(kToPeers && kSwiGLUQuant) &&
                    !(kMany && (kSwiGLUQuant || kFromStaging)),
                "unsupported form");
  constexpr int kHalves = kSwiGLUQuant ? 2 : 1;
  using S = Shape<kHalves>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  Control* ctl = reinterpret_cast<Control*>(ring + g.ring_bytes);
  // (kToPeers only) behind the control block; the tables come last.
  using Peers = PeerStage<kPeerTokens>;
  Peers* peer_stage = reinterpret_cast<Peers*>(ctl + 1);
  uint32_t* tile_start = kToPeers ? reinterpret_cast<uint32_t*>(peer_stage + 1)
                                  : reinterpret_cast<uint32_t*>(ctl + 1);  // [E + 1]
  uint32_t* rows_of = tile_start + g.num_experts + 1;                      // [E] valid rows
  uint32_t* a_row0 = rows_of + g.num_experts;  // [E] first row in the token plane
  uint32_t* src_rows =                         // [E][world] or null
      (kFromStaging && g.src_table != 0) ? a_row0 + g.num_experts : nullptr;
  const A2AParams& p = g.a2a;
  int parity = 0;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile uint32_t* abort_flag = &ctl->abort_flag;
  const int w_blocks = ceil_div<int>(g.n_out, 128);
  const int num_kb = ceil_div<int>(g.k, kBlockKBytes);

  if (tid == 0) {
    ctl->abort_flag = 0;
    ctl->max_tokens = 16;
    for (int s = 0; s < kMaxStages; ++s) {
      tc::mbar_init(&ctl->full[s], 1);
      tc::mbar_init(&ctl->empty[s], 1);
    }
    for (int b = 0; b < kBuffers; ++b) {
      tc::mbar_init(&ctl->part_full[b], 2);  // the MMAs, and the scales
      tc::mbar_init(&ctl->part_empty[b], 8);
    }
    if constexpr (kMany) rows::init_barriers(&ctl->row_bar);
    tc::fence_mbar_init();
    tc::tma_prefetch_desc(&tmap_w);
    tc::tma_prefetch_desc(&tmap_x64);
    tc::tma_prefetch_desc(&tmap_x16);
  }
  if (warp == 2) {
    tc::tmem_alloc(&ctl->tmem_base, kTmemCols);
    tc::tmem_relinquish();
  }
  ptx::wait_for_previous_kernels();
  if constexpr (!kFromStaging) ptx::let_next_kernel_start();
  if constexpr (kFromStaging || kToPeers) parity = static_cast<int>(ptx::ld_volatile(p.iter) & 1u);
  if constexpr (kFromStaging) {
    // Role of the dispatch receive phase: rows per (source, expert) from the posted
    // histograms, the layout of the packed staging, the per-expert totals.
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
    for (int le = tid; le < g.num_experts; le += blockDim.x) a_row0[le] = rows_of[le];
    __syncthreads();
    if (warp == 0) warp_exclusive_scan_smem(a_row0, g.num_experts, lane, false);
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
      a_row0[e] = 0;
    }
    rows_of[e] = static_cast<uint32_t>(rows);
    const int tiles = token_tiles(rows, S::kMaxTokens);
    tile_start[e] = static_cast<uint32_t>(tiles * w_blocks);
    if (tiles > 0) atomicMax(&ctl->max_tokens, static_cast<uint32_t>(token_width(rows, tiles)));
  }
  if constexpr (kToPeers) {
    if (blockIdx.x == 0) {
      // Role of the combine send phase's first block: the dispatch that produced these
      // rows is over on this rank, so clear its flag set and move on.
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
  if (warp == 0) warp_exclusive_scan_smem(tile_start, g.num_experts, lane, true);
  tc::tc_fence_before_sync();
  __syncthreads();
  tc::tc_fence_after_sync();
  const uint32_t tmem_base = ctl->tmem_base;
  const uint32_t total_tiles = tile_start[g.num_experts];
  // As many stages as the launch's widest token tile leaves room for.
  const uint32_t stage_bytes = S::kWBytes + ctl->max_tokens * kBlockKBytes;
  const uint32_t stages = min(g.ring_bytes / stage_bytes, static_cast<uint32_t>(kMaxStages));
  if constexpr (kMany) {
    const rows::Shared shared{ring,       &ctl->row_bar, &ctl->seg[0][0][0][0], peer_stage,
                              tile_start, rows_of,       abort_flag,            tmem_base};
    rows::run<kToPeers>(tmap_w, tmap_x64, g, shared);
  } else if (warp == 0) {
    if (tc::elect_one()) {
      uint32_t stage = 0, phase = 0, pending = 0, pending_phase = 0;
      bool ok = *abort_flag == 0u;
      int last_expert = -1;  // expert that `landed` refers to
      uint32_t landed = 0;   // bit s: the rows of source s for that expert have landed
      for (uint32_t t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
        const Tile c = locate<kHalves>(tile_start, rows_of, g.num_experts, t);
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
        const int x_row = static_cast<int>(a_row0[c.expert]) + c.first;
        const int x_plane = kFromStaging ? 0 : c.expert;
        const uint32_t tx = S::kWBytes + static_cast<uint32_t>(c.width) * kBlockKBytes;
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = tc::mbar_wait(&ctl->empty[stage], phase ^ 1u, abort_flag, kWaitLimitNs);
          if (!ok) break;
          uint8_t* w_dst = ring + stage * stage_bytes;
          uint8_t* x_dst = w_dst + S::kWBytes;
          tc::mbar_arrive_expect_tx(&ctl->full[stage], tx);
          pending |= 1u << stage;
          pending_phase = (pending_phase & ~(1u << stage)) | (phase << stage);
          tc::tma_load_3d(w_dst, &tmap_w, &ctl->full[stage], kb * kBlockKBytes, c.w_blk * 128,
                          c.expert);
          if constexpr (kHalves == 2)
            tc::tma_load_3d(w_dst + kBlockM * kBlockKBytes, &tmap_w, &ctl->full[stage],
                            kb * kBlockKBytes, g.n_out + c.w_blk * 128, c.expert);
          int r = 0;
          for (; r + 64 <= c.width; r += 64)
            tc::tma_load_3d(x_dst + r * kBlockKBytes, &tmap_x64, &ctl->full[stage],
                            kb * kBlockKBytes, x_row + r, x_plane);
          for (; r < c.width; r += 16)
            tc::tma_load_3d(x_dst + r * kBlockKBytes, &tmap_x16, &ctl->full[stage],
                            kb * kBlockKBytes, x_row + r, x_plane);
          if (++stage == stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      // (The scales' warp waits for the same rows, which have all landed.)
      if constexpr (kFromStaging) ptx::let_next_kernel_start();
      if (!ok || *abort_flag != 0u) {
        const uint64_t t0 = ptx::globaltimer_ns();
        for (uint32_t s = 0; s < stages; ++s) {
          if (!((pending >> s) & 1u)) continue;
          while (!tc::mbar_try_wait(&ctl->full[s], (pending_phase >> s) & 1u)) {
            if (ptx::globaltimer_ns() - t0 > 100000000ull) break;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (tc::elect_one()) {
      uint32_t stage = 0, phase = 0, round = 0;
      bool ok = *abort_flag == 0u;
      for (uint32_t t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
        const Tile c = locate<kHalves>(tile_start, rows_of, g.num_experts, t);
        // kind::f8f6f4, e4m3 x e4m3 -> f32.
        const uint32_t idesc = tc::make_instr_desc(0u, kBlockM, c.width);
        for (int kb = 0; kb < num_kb && ok; ++kb, ++round) {
          const uint32_t buf = round % kBuffers;
          ok = tc::mbar_wait(&ctl->part_empty[buf], ((round / kBuffers) & 1u) ^ 1u, abort_flag,
                             kWaitLimitNs) &&
               tc::mbar_wait(&ctl->full[stage], phase, abort_flag, kWaitLimitNs);
          if (!ok) break;
          tc::tc_fence_after_sync();
          const uint8_t* w_src = ring + stage * stage_bytes;
          const uint64_t x_desc = tc::make_smem_desc_sw128(w_src + S::kWBytes);
#pragma unroll
          for (int h = 0; h < kHalves; ++h) {
            const uint64_t w_desc = tc::make_smem_desc_sw128(w_src + h * kBlockM * kBlockKBytes);
#pragma unroll
            for (int k = 0; k < kBlockKBytes / kUmmaKBytes; ++k) {
              tc::mma_f8_ss(tmem_base + buf * 128 + h * S::kMaxTokens,
                            tc::advance_smem_desc(w_desc, k * kUmmaKBytes),
                            tc::advance_smem_desc(x_desc, k * kUmmaKBytes), idesc, k != 0);
            }
          }
          tc::mma_commit(&ctl->empty[stage]);
          tc::mma_commit(&ctl->part_full[buf]);
          if (++stage == stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 3) {
    // Products of the scales.  Lane l owns tokens l, l + 32, ... of the tile.
    constexpr int kOwn = S::kMaxTokens / 32;
    constexpr int kChunk = 4;  // K blocks whose scales are fetched together, a chunk ahead
    uint32_t round = 0;
    bool ok = *abort_flag == 0u;
    int last_expert = -1;
    uint32_t landed = 0;  // (lane 0)
    for (uint32_t t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
      const Tile c = locate<kHalves>(tile_start, rows_of, g.num_experts, t);
      if constexpr (kFromStaging) {
        // The scales sit behind the rows in the staging that peers write: wait for the same
        // sources as the TMA producer does (lane 0 acquires, the warp follows).
        if (c.expert != last_expert) {
          last_expert = c.expert;
          landed = 0;
        }
        int good = 1;
        if (lane == 0)
          good = wait_tile_sources(p, c.expert, c.first, min(c.first + c.width, c.rows), parity,
                                   src_rows, landed)
                     ? 1
                     : 0;
        good = __shfl_sync(0xffffffffu, good, 0);
        __syncwarp();
        if (good == 0) {
          if (lane == 0) *abort_flag = 1u;
          ok = false;
          break;
        }
      }
      const float* sa_row[kOwn];
#pragma unroll
      for (int i = 0; i < kOwn; ++i) {
        const int row = c.first + lane + 32 * i;
        const int safe = row < c.rows ? row : c.first;
        if constexpr (kFromStaging) {
          sa_row[i] = reinterpret_cast<const float*>(
              p.peer[p.rank] + p.off_disp_stage +
              (static_cast<size_t>(a_row0[c.expert]) + safe) * p.slot_bytes + p.hidden_bytes);
        } else {
          sa_row[i] = g.sa + c.expert * g.sa_stride_e + safe * g.sa_stride_row;
        }
      }
      const float* sw0 = g.sw + c.expert * g.sw_stride_e + c.w_blk * g.sw_stride_row;
      const float* sw1 = sw0 + (g.n_out / 128) * g.sw_stride_row;  // kHalves == 2
      float a[kChunk][kOwn], a_next[kChunk][kOwn], w[kChunk][2], w_next[kChunk][2];
      auto fetch = [&](int kb0) {
#pragma unroll
        for (int u = 0; u < kChunk; ++u) {
          const int kb = min(kb0 + u, num_kb - 1);
#pragma unroll
          for (int i = 0; i < kOwn; ++i) {
            if (lane + 32 * i < c.width)
              a_next[u][i] = kFromStaging ? __ldcg(sa_row[i] + kb) : __ldg(sa_row[i] + kb);
          }
          w_next[u][0] = __ldg(sw0 + kb);
          if constexpr (kHalves == 2) w_next[u][1] = __ldg(sw1 + kb);
        }
      };
      fetch(0);
      for (int kb0 = 0; kb0 < num_kb && ok; kb0 += kChunk) {
#pragma unroll
        for (int u = 0; u < kChunk; ++u) {
#pragma unroll
          for (int i = 0; i < kOwn; ++i) a[u][i] = a_next[u][i];
          w[u][0] = w_next[u][0];
          w[u][1] = w_next[u][1];
        }
        if (kb0 + kChunk < num_kb) fetch(kb0 + kChunk);
#pragma unroll
        for (int u = 0; u < kChunk; ++u) {
          if (kb0 + u >= num_kb || !ok) continue;
          const uint32_t buf = round % kBuffers;
          ok = tc::mbar_wait(&ctl->part_empty[buf], ((round / kBuffers) & 1u) ^ 1u, abort_flag,
                             kWaitLimitNs);
          ++round;
          if (!ok) continue;
#pragma unroll
          for (int i = 0; i < kOwn; ++i) {
            const int n = lane + 32 * i;
            if (n < c.width) {
#pragma unroll
              for (int h = 0; h < kHalves; ++h)
                ctl->scales[buf][h * S::kMaxTokens + n] = a[u][i] * w[u][h];
            }
          }
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&ctl->part_full[buf]);
        }
      }
    }
  } else if (warp >= 4) {
    const int ew = (warp - 4) & 3;  // tensor-memory lanes [32 * ew, +32)
    const int wg = (warp - 4) >> 2;  // 16-token groups wg, wg + 2, wg + 4, ...
    const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(ew * 32) << 16);
    uint32_t round = 0;
    uint32_t pending_signals = 0;  // kToPeers, warp 4: queued arrival adds
    bool ok = *abort_flag == 0u;
    for (uint32_t t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
      const Tile c = locate<kHalves>(tile_start, rows_of, g.num_experts, t);
      const int groups = c.width >> 4;
      const int live = min(c.width, c.rows - c.first);  // tokens of the tile that exist
      Group acc[kHalves][S::kGroups];
      const int own_groups = (groups - wg + 1) >> 1;  // of this warp group
      const FoldLoop loop{ctl, abort_flag, t_lane, num_kb, wg, lane};
      ok = fold_tile<kHalves>(loop, own_groups, acc, round);
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

      const int n_tid = tid - 128;  // 0..255 over the eight warps
      // ---- tile epilogue ------------------------------------------------------
      if constexpr (kFromStaging) {
        // The first block of columns also records where the rows came from.
        if (c.w_blk == 0 && n_tid < live) {
          const int row = c.first + n_tid;
          const uint8_t* slot = p.peer[p.rank] + p.off_disp_stage +
                                (static_cast<size_t>(a_row0[c.expert]) + row) * p.slot_bytes;
          const int4 tr = ptx::ld_cg_v4(slot + p.trailer_off);
          uint2 rs;
          rs.x = (static_cast<uint32_t>(tr.w) & 0xffffu) | (static_cast<uint32_t>(tr.y) << 16);
          rs.y = static_cast<uint32_t>(tr.x);
          p.row_src[static_cast<size_t>(c.expert) * p.cap + row] = rs;
        }
      }
      const int lt = n_tid & 127;  // thread of the warp group
      if constexpr (kToPeers) {
        // Where each token's row goes, and whose token it is.
        if (n_tid < c.width) {
          unsigned long long off = 0;
          uint32_t sig_token = kNoSignal, sig_group = 0;
          if (n_tid < live) {
            const uint2 rs = p.row_src[static_cast<size_t>(c.expert) * p.cap + c.first + n_tid];
            const int src_rank = static_cast<int>(rs.x & 0xffffu);
            const uint32_t k = rs.x >> 16;
            const uint32_t token = rs.y;
            if (token < static_cast<uint32_t>(p.max_tokens) && k < static_cast<uint32_t>(p.topk) &&
                src_rank < p.world) {
              sig_token = token;
              sig_group = static_cast<uint32_t>((src_rank / p.dp_size) * p.dp_size);
              off = p.off_comb_stage +
                    (static_cast<size_t>(token) * p.topk + k) * (static_cast<size_t>(g.n_out) * 2);
            } else {
              report_failure(p.status, kBadToken, kPhaseCombinePayload, src_rank, p.max_tokens,
                             token, p.rank);
            }
          }
          peer_stage->token[n_tid] = sig_token;
          peer_stage->group[n_tid] = sig_group;
          peer_stage->row_off[n_tid] = off;
        }
        asm volatile("bar.sync 4, 256;" ::: "memory");
      }
      if constexpr (kSwiGLUQuant) {
        // acc[0] = gate, acc[1] = up; the 128 columns of the tile are one scale block of each
        // token.  The result replaces the gate sums.
#pragma unroll
        for (int i = 0; i < S::kGroups; ++i) {
          if (2 * i + wg >= groups) continue;
          float m[4] = {0.f, 0.f, 0.f, 0.f};  // tokens {0, 1} and {8, 9} + 2 * (lane % 4)
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float2 v = unpack2(acc[0][i].pair[j]);
            const float2 u = unpack2(acc[1][i].pair[j]);
            v.x = silu(v.x) * u.x;
            v.y = silu(v.y) * u.y;
            acc[0][i].pair[j] = pack2(__float_as_uint(v.x), __float_as_uint(v.y));
            m[2 * (j & 1)] = fmaxf(m[2 * (j & 1)], fabsf(v.x));
            m[2 * (j & 1) + 1] = fmaxf(m[2 * (j & 1) + 1], fabsf(v.y));
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) {
#pragma unroll
            for (int o = 4; o <= 16; o <<= 1)
              m[q] = fmaxf(m[q], __shfl_xor_sync(0xffffffffu, m[q], o));
          }
          if (lane < 4) {
            float* dst = &ctl->amax[wg][ew][i * 16 + 2 * lane];
            *reinterpret_cast<float2*>(dst) = make_float2(m[0], m[1]);
            *reinterpret_cast<float2*>(dst + 8) = make_float2(m[2], m[3]);
          }
        }
        sync_group(wg);
        if (lt < 16 * S::kGroups) {
          const float(*amax)[64] = ctl->amax[wg];
          const float m = fmaxf(fmaxf(fmaxf(amax[0][lt], amax[1][lt]),
                                      fmaxf(amax[2][lt], amax[3][lt])), 1e-4f);
          const float scale = m / 448.0f;
          ctl->inv_scale[wg][lt] = 1.0f / scale;
          const int n = (2 * (lt >> 4) + wg) * 16 + (lt & 15);
          if (n < live)
            g.out_scale[c.expert * g.os_stride_e +
                        static_cast<int64_t>(c.first + n) * g.os_stride_row + c.w_blk] = scale;
        }
        sync_group(wg);
      }
      // A thread's values lie across token rows; each group passes through shared memory so that
      // rows leave in 16-byte pieces.
#pragma unroll
      for (int i = 0; i < S::kGroups; ++i) {
        const int grp = 2 * i + wg;
        if (grp >= groups) continue;
        uint8_t(*seg)[kSegBytes] = ctl->seg[wg][i & 1];
        if constexpr (kSwiGLUQuant) {
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            const int t0 = 8 * b + 2 * (lane & 3);
            const float2 inv = *reinterpret_cast<const float2*>(&ctl->inv_scale[wg][i * 16 + t0]);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const float2 v = unpack2(acc[0][i].pair[2 * q + b]);
              const uint32_t e = __nv_cvt_float2_to_fp8x2(make_float2(v.x * inv.x, v.y * inv.y),
                                                          __NV_SATFINITE, __NV_E4M3);
              uint8_t* dst = &seg[t0][ew * 32 + 8 * q + (lane >> 2)];
              dst[0] = static_cast<uint8_t>(e);
              dst[kSegBytes] = static_cast<uint8_t>(e >> 8);
            }
          }
          sync_group(wg);
          const int n = grp * 16 + (lt >> 3);
          if (n < live)
            *reinterpret_cast<int4*>(static_cast<uint8_t*>(g.out) + c.expert * g.out_stride_e +
                                     static_cast<int64_t>(c.first + n) * g.out_stride_row +
                                     c.w_blk * 128 + (lt & 7) * 16) =
                *reinterpret_cast<const int4*>(&seg[lt >> 3][(lt & 7) * 16]);
        } else {
#pragma unroll
          for (int b = 0; b < 2; ++b)
            stmatrix_x4_trans(&seg[8 * b + (lane & 7)][(ew * 32 + (lane >> 3) * 8) * 2],
                              bf16_pair(acc[0][i].pair[b]), bf16_pair(acc[0][i].pair[2 + b]),
                              bf16_pair(acc[0][i].pair[4 + b]), bf16_pair(acc[0][i].pair[6 + b]));
          sync_group(wg);
          const int col = c.w_blk * 128 + (lt & 15) * 8;
#pragma unroll
          for (int it = 0; it < 2; ++it) {
            const int tok = it * 8 + (lt >> 4);
            const int n = grp * 16 + tok;
            const int4 v = *reinterpret_cast<const int4*>(&seg[tok][(lt & 15) * 16]);
            if (col + 8 > g.n_out) continue;
            if constexpr (kToPeers) {
              if (peer_stage->token[n] != kNoSignal) {
                const uint32_t first_rank = peer_stage->group[n];
                const size_t off = peer_stage->row_off[n] + static_cast<size_t>(col) * 2;
                for (int r = 0; r < min(p.dp_size, 8); ++r) ptx::st_v4(p.peer[first_rank + r] + off, v);
              }
            } else if (n < live) {
              *reinterpret_cast<int4*>(static_cast<__nv_bfloat16*>(g.out) +
                                       c.expert * g.out_stride_e +
                                       static_cast<int64_t>(c.first + n) * g.out_stride_row + col) = v;
            }
          }
        }
      }
      if constexpr (kToPeers) {
        // Arrival is counted in columns: this tile's share of each row.  The adds are queued
        // and flushed behind ONE system-scope fence for as many tiles as the queue holds: with a
        // handful of rows per expert a fence per tile would cost more than the tile.
        asm volatile("bar.sync 4, 256;" ::: "memory");
        if (warp == 4) {
          const uint32_t units = static_cast<uint32_t>(min(128, g.n_out - c.w_blk * 128));
          if (pending_signals + c.width > kQueue) {
            flush(p, peer_stage, pending_signals, lane);
            pending_signals = 0;
          }
          for (int j0 = 0; j0 < c.width; j0 += 32) {
            const uint32_t tok = j0 + lane < c.width ? peer_stage->token[j0 + lane] : kNoSignal;
            const bool there = tok != kNoSignal;
            const uint32_t mask = __ballot_sync(0xffffffffu, there);
            if (there) {
              const uint32_t at = pending_signals + __popc(mask & ((1u << lane) - 1u));
              peer_stage->q_token[at] = tok;
              peer_stage->q_group_units[at] = peer_stage->group[j0 + lane] | (units << 8);
            }
            pending_signals += __popc(mask);
          }
        }
        // (The barrier at the top of the next tile's epilogue comes before the token table is
        // rewritten.)
      }
    }
    if constexpr (kToPeers) {
      // What is still queued (also after a failed wait: rows that were stored are announced).
      if (warp == 4 && pending_signals > 0) flush(p, peer_stage, pending_signals, lane);
    }
  }

  tc::tc_fence_before_sync();
  __syncthreads();
  if (warp == 2) {
    tc::tc_fence_after_sync();
    tc::tmem_dealloc(tmem_base, kTmemCols);
  }
  if (tid == 0 && ctl->abort_flag != 0u && g.status != nullptr) atomicMax(g.status, 1u);
  (void)parity;
}

}  // namespace fold
}  // namespace
}  // namespace pplx
