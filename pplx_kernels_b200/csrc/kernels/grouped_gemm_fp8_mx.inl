// fp8 expert GEMM with power-of-two scales (included by grouped_gemm_fp8_sm100.cu): the tensor
// cores apply the scales (kind::mxf8f6f4.block_scale) and the whole K range accumulates in tensor
// memory.
//
// As in the form with fp32 scales the WEIGHTS are the M operand and the tokens the N operand: a
// tile is 256 weight rows, as two MMAs of M = 128 (SwiGLU: 128 gate and 128 up rows, one scale
// block of the result), times a token tile of 16 to 224 rows of one expert.  Both halves read the
// same tokens, so at the full width a stage moves 60 KB for 900 cycles of MMAs, within what L2
// gives an SM; with 128 tokens as M and 256 weight rows as N it was 48 KB for 512, and an expert
// was padded to 128 rows.  Where no token tile is wider than 112 rows there are two accumulators
// and the epilogue of a tile runs under the MMAs of the next.
//
// Layers before and after: Qwen3-30B-A3B (128 experts of 768 x 2048) with 61 tokens 183.5 -> 143
// us, 1000 tokens 203 -> 172 us, 4000 tokens 389 -> 355 us; DeepSeek-V2-Lite (64 of 1408 x 2048)
// with 300 tokens 189 -> 137 us, 4000 tokens 412 -> 367 us; Mixtral 8x7B (8 of 14336 x 4096) with
// 64 tokens 282 -> 256 us, 700 tokens 399 -> 370 us, 2048 and 4096 tokens level (785, 1414 us).
//
// Roles: warp 0 TMA producer, warp 1 MMA issuer, warp 2 tensor-memory allocation, warp 3
// scales, warps 4-11 epilogue.
namespace pplx {
namespace {
namespace mx {

using namespace tok;

constexpr int kMaxStages = 6;
constexpr int kMaxTokens = 224;
constexpr int kHalfTokens = kMaxTokens / 2;
constexpr uint32_t kWBytes = 2 * kBlockM * kBlockKBytes;
constexpr uint32_t kScaleCol = 2 * kMaxTokens;  // weights of both halves, tokens, tokens from 128
constexpr uint32_t kAtomBytes = 512;            // scales of 128 rows for one K block
constexpr int kBatch = 3;                       // 16-token groups that an epilogue warp reads at once
constexpr int kSegBytes = 256 + 16;             // 128 columns of bf16 of one token, padded
constexpr int kSegBytesQ = 128 + 16;            // 128 columns of e4m3
constexpr int kSegArea = 2 * 16 * kSegBytes;
static_assert(kBatch * 16 * kSegBytesQ <= kSegArea, "SwiGLU staging");

struct Tile {
  int expert;
  int w_blk;    // block of output columns
  int first;    // first token row of the tile inside its expert
  int width;    // token rows of the tile, a multiple of 16
  int rows;     // valid rows of the expert
};

struct Control {
  uint64_t full[kMaxStages];
  uint64_t empty[kMaxStages];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  uint32_t abort_flag;
  uint32_t max_tokens;                           // widest token tile of this launch
  uint32_t pad;
  alignas(16) float amax[2][4][kBatch * 16];     // SwiGLU: [warp group][warp][token]
  // [warp group], then plain: [alternating][16 tokens][kSegBytes], SwiGLU: [kBatch * 16 tokens]
  // [kSegBytesQ].
  alignas(16) uint8_t seg[2][kSegArea];
  alignas(128) uint8_t sf[kMaxStages][4 * kAtomBytes];
};

// Tiles of an expert are ordered with the token tile fastest: CTAs that run at the same time
// share a block of weights in L2.
__device__ __forceinline__ Tile locate(const uint32_t* tile_start, const uint32_t* rows_of,
                                       int num_experts, uint32_t t) {
  Tile c;
  c.expert = find_group(tile_start, num_experts, t);
  c.rows = static_cast<int>(rows_of[c.expert]);
  const int tiles = token_tiles(c.rows, kMaxTokens);
  const uint32_t rem = t - tile_start[c.expert];
  c.w_blk = static_cast<int>(rem / tiles);
  c.width = token_width(c.rows, tiles);
  c.first = static_cast<int>(rem - static_cast<uint32_t>(c.w_blk) * tiles) * c.width;
  return c;
}

// E8M0 byte of a power-of-two fp32 scale (its exponent field), for all four K steps.
__device__ __forceinline__ uint32_t e8m0_x4(float scale) {
  return ((__float_as_uint(scale) >> 23) & 0xffu) * 0x01010101u;
}

// The smallest power of two that is not below v (v > 0, finite).
__device__ __forceinline__ float pow2_not_below(float v) {
  const uint32_t bits = __float_as_uint(v);
  const uint32_t exp = (bits >> 23) + ((bits & 0x7fffffu) != 0u ? 1u : 0u);
  return __uint_as_float(exp << 23);
}

__device__ __forceinline__ uint32_t bf16_bits(uint32_t a, uint32_t b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(a), __uint_as_float(b));
  return *reinterpret_cast<const uint32_t*>(&h);
}

template <bool kSwiGLUQuant, bool kFromStaging, bool kToPeers>
__global__ void __launch_bounds__(kThreads, 1)
    grouped_gemm_fp8_mx_kernel(const __grid_constant__ CUtensorMap tmap_w,
                                 const __grid_constant__ CUtensorMap tmap_x64,
                                 const __grid_constant__ CUtensorMap tmap_x16,
                                 const __grid_constant__ Fp8GemmArgs g) {
  static_assert(!(kFromStaging && kToPeers) && !(kToPeers && kSwiGLUQuant), "unsupported form");
  constexpr int kCols = kSwiGLUQuant ? 128 : 256;  // output columns of a tile
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
  const int w_blocks = ceil_div<int>(g.n_out, kCols);
  const int num_kb = ceil_div<int>(g.k, kBlockKBytes);

  if (tid == 0) {
    ctl->abort_flag = 0;
    ctl->max_tokens = 16;
    for (int s = 0; s < kMaxStages; ++s) {
      tc::mbar_init(&ctl->full[s], 2);  // the bytes, and the scales
      tc::mbar_init(&ctl->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(&ctl->acc_full[b], 1);
      tc::mbar_init(&ctl->acc_empty[b], 8);
    }
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
    const int tiles = token_tiles(rows, kMaxTokens);
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
  const uint32_t stage_bytes = kWBytes + ctl->max_tokens * kBlockKBytes;
  const uint32_t stages = min(g.ring_bytes / stage_bytes, static_cast<uint32_t>(kMaxStages));
  // Two accumulators where two of the widest token tile fit.
  const uint32_t buffers = ctl->max_tokens <= kHalfTokens ? 2u : 1u;
  const uint32_t half_cols = buffers == 2u ? kHalfTokens : kMaxTokens;
  if (warp == 0) {
    if (tc::elect_one()) {
      uint32_t stage = 0, phase = 0, pending = 0, pending_phase = 0;
      bool ok = *abort_flag == 0u;
      int last_expert = -1;  // expert that `landed` refers to
      uint32_t landed = 0;   // bit s: the rows of source s for that expert have landed
      for (uint32_t t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
        const Tile c = locate(tile_start, rows_of, g.num_experts, t);
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
        const uint32_t tx = kWBytes + static_cast<uint32_t>(c.width) * kBlockKBytes;
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = tc::mbar_wait(&ctl->empty[stage], phase ^ 1u, abort_flag, kWaitLimitNs);
          if (!ok) break;
          uint8_t* w_dst = ring + stage * stage_bytes;
          uint8_t* x_dst = w_dst + kWBytes;
          tc::mbar_arrive_expect_tx(&ctl->full[stage], tx);
          pending |= 1u << stage;
          pending_phase = (pending_phase & ~(1u << stage)) | (phase << stage);
          tc::tma_load_3d(w_dst, &tmap_w, &ctl->full[stage], kb * kBlockKBytes, c.w_blk * kCols,
                          c.expert);
          tc::tma_load_3d(w_dst + kBlockM * kBlockKBytes, &tmap_w, &ctl->full[stage],
                          kb * kBlockKBytes,
                          kSwiGLUQuant ? g.n_out + c.w_blk * 128 : c.w_blk * 256 + 128, c.expert);
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
      uint32_t stage = 0, phase = 0, local = 0;
      bool ok = *abort_flag == 0u;
      for (uint32_t t = blockIdx.x; t < total_tiles && ok; t += gridDim.x, ++local) {
        const Tile c = locate(tile_start, rows_of, g.num_experts, t);
        const uint32_t buf = local % buffers, use = local / buffers;
        ok = tc::mbar_wait(&ctl->acc_empty[buf], (use & 1u) ^ 1u, abort_flag, kWaitLimitNs);
        if (!ok) break;
        tc::tc_fence_after_sync();
        const uint32_t tmem_d = tmem_base + buf * kMaxTokens;
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = tc::mbar_wait(&ctl->full[stage], phase, abort_flag, kWaitLimitNs);
          if (!ok) break;
          tc::tc_fence_after_sync();
          const uint8_t* w_src = ring + stage * stage_bytes;
          const uint64_t x_desc = tc::make_smem_desc_sw128(w_src + kWBytes);
          // (Ordered with this thread's MMAs before and after: one set of columns is enough.)
          const uint8_t* sf = ctl->sf[stage];
#pragma unroll
          for (int a = 0; a < 3; ++a)
            tc::tmem_cp_32x128b_warpx4(tmem_base + kScaleCol + 4 * a,
                                       tc::make_smem_desc_rows16(sf + a * kAtomBytes));
          if (c.width > 128)
            tc::tmem_cp_32x128b_warpx4(tmem_base + kScaleCol + 12,
                                       tc::make_smem_desc_rows16(sf + 3 * kAtomBytes));
#pragma unroll
          for (uint32_t h = 0; h < 2; ++h) {
            const uint64_t w_desc = tc::make_smem_desc_sw128(w_src + h * kBlockM * kBlockKBytes);
#pragma unroll
            for (uint32_t k = 0; k < kBlockKBytes / kUmmaKBytes; ++k) {
              tc::mma_mxf8_ss(tmem_d + h * half_cols, tc::advance_smem_desc(w_desc, k * kUmmaKBytes),
                              tc::advance_smem_desc(x_desc, k * kUmmaKBytes),
                              tc::make_instr_desc_mxf8(kBlockM, c.width, k),
                              (tmem_base + kScaleCol + 4 * h) | (k << 30),
                              (tmem_base + kScaleCol + 8) | (k << 30), kb != 0 || k != 0);
            }
          }
          tc::mma_commit(&ctl->empty[stage]);
          if (++stage == stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (ok) tc::mma_commit(&ctl->acc_full[buf]);
      }
    }
    __syncwarp();
  } else if (warp == 3) {
    // The scales of each K block as E8M0 bytes, where tcgen05.cp finds them: an atom is 32 rows
    // of 16 bytes, row l holding rows (tokens) l, l + 32, l + 64 and l + 96, a byte for each
    // K = 32 step.  Two atoms of the weights, whose 128 rows share a scale, two of the tokens.
    constexpr int kOwn = kMaxTokens / 32;
    constexpr int kChunk = 4;  // K blocks whose scales are fetched together, a chunk ahead
    uint32_t stage = 0, phase = 0;
    bool ok = *abort_flag == 0u;
    uint32_t not_pow2 = 0;  // mantissa bits seen in any scale: the caller's promise was broken
    int last_expert = -1;
    uint32_t landed = 0;  // (lane 0)
    const int last_block = (((kSwiGLUQuant ? 2 : 1) * g.n_out) - 1) / 128;
    for (uint32_t t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
      const Tile c = locate(tile_start, rows_of, g.num_experts, t);
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
      bool live[kOwn];
#pragma unroll
      for (int i = 0; i < kOwn; ++i) {
        live[i] = lane + 32 * i < c.width && c.first + lane + 32 * i < c.rows;
        const int row = live[i] ? c.first + lane + 32 * i : 0;
        if constexpr (kFromStaging) {
          sa_row[i] = reinterpret_cast<const float*>(
              p.peer[p.rank] + p.off_disp_stage +
              (static_cast<size_t>(a_row0[c.expert]) + row) * p.slot_bytes + p.hidden_bytes);
        } else {
          sa_row[i] = g.sa + c.expert * g.sa_stride_e + row * g.sa_stride_row;
        }
      }
      const int blk0 = kSwiGLUQuant ? c.w_blk : 2 * c.w_blk;
      const int blk1 = kSwiGLUQuant ? g.n_out / 128 + c.w_blk : blk0 + 1;
      const float* sw0 = g.sw + c.expert * g.sw_stride_e + min(blk0, last_block) * g.sw_stride_row;
      const float* sw1 = g.sw + c.expert * g.sw_stride_e + min(blk1, last_block) * g.sw_stride_row;
      float a[kChunk][kOwn], a_next[kChunk][kOwn], w[kChunk][2], w_next[kChunk][2];
      auto fetch = [&](int kb0) {
#pragma unroll
        for (int u = 0; u < kChunk; ++u) {
          const int kb = min(kb0 + u, num_kb - 1);
#pragma unroll
          for (int i = 0; i < kOwn; ++i) {
            // (Rows that do not exist: 2^0; their results are not stored.)
            a_next[u][i] = 1.0f;
            if (live[i]) a_next[u][i] = kFromStaging ? __ldcg(sa_row[i] + kb) : __ldg(sa_row[i] + kb);
          }
          w_next[u][0] = __ldg(sw0 + kb);
          w_next[u][1] = __ldg(sw1 + kb);
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
          ok = tc::mbar_wait(&ctl->empty[stage], phase ^ 1u, abort_flag, kWaitLimitNs);
          if (!ok) continue;
          auto* atoms = reinterpret_cast<uint4*>(ctl->sf[stage]) + lane;
          constexpr int kAtom = kAtomBytes / 16;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            not_pow2 |= __float_as_uint(w[u][h]) & 0x7fffffu;
            const uint32_t b = e8m0_x4(w[u][h]);
            atoms[h * kAtom] = make_uint4(b, b, b, b);
          }
          uint32_t e[8];
          e[7] = 0;
#pragma unroll
          for (int i = 0; i < kOwn; ++i) {
            not_pow2 |= __float_as_uint(a[u][i]) & 0x7fffffu;
            e[i] = e8m0_x4(a[u][i]);
          }
          atoms[2 * kAtom] = make_uint4(e[0], e[1], e[2], e[3]);
          if (c.width > 128) atoms[3 * kAtom] = make_uint4(e[4], e[5], e[6], e[7]);
          ptx::fence_proxy_async_smem();  // these writes, before tcgen05.cp reads them
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&ctl->full[stage]);
          if (++stage == stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    }
    if (__any_sync(0xffffffffu, not_pow2 != 0u) && lane == 0 && g.status != nullptr)
      atomicMax(g.status, 2u);
  } else if (warp >= 4) {
    const int ew = (warp - 4) & 3;  // tensor-memory lanes [32 * ew, +32)
    const int wg = (warp - 4) >> 2;  // 16-token groups wg, wg + 2, wg + 4, ...
    const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(ew * 32) << 16);
    uint32_t local = 0;
    uint32_t pending_signals = 0;  // kToPeers, warp 4: queued arrival adds
    bool ok = *abort_flag == 0u;
    for (uint32_t t = blockIdx.x; t < total_tiles && ok; t += gridDim.x, ++local) {
      const Tile c = locate(tile_start, rows_of, g.num_experts, t);
      const int groups = c.width >> 4;
      const int live = min(c.width, c.rows - c.first);  // tokens of the tile that exist
      const uint32_t buf = local % buffers, use = local / buffers;
      ok = tc::mbar_wait(&ctl->acc_full[buf], use & 1u, abort_flag, kWaitLimitNs);
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
      // A thread's values lie across token rows; each group of 16 tokens passes through shared
      // memory so that rows leave in 16-byte pieces.  kBatch groups are read at once, and the
      // accumulator is handed back when the last of them are in registers: with one accumulator
      // the MMAs of the next tile wait for that.
      const uint32_t t_acc = t_lane + buf * kMaxTokens;
      auto hand_back = [&] {
        tc::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&ctl->acc_empty[buf]);
      };
      if (wg >= groups) hand_back();
      int alt = 0;
#pragma unroll 1
      for (int g0 = wg; g0 < groups; g0 += 2 * kBatch) {
        const bool last = g0 + 2 * kBatch >= groups;
        if constexpr (kSwiGLUQuant) {
          // The first half of the accumulator is gate, the second up; the 128 columns of the
          // tile are one scale block of each token.
          float r[kBatch][2][8];
#pragma unroll
          for (int i = 0; i < kBatch; ++i) {
            if (g0 + 2 * i >= groups) break;
            uint32_t v[2][8], up[2][8];
            load_group(t_acc + (g0 + 2 * i) * 16, v[0], v[1]);
            load_group(t_acc + half_cols + (g0 + 2 * i) * 16, up[0], up[1]);
            tc::tmem_ld_wait();
#pragma unroll
            for (int q = 0; q < 2; ++q) {
#pragma unroll
              for (int j = 0; j < 8; ++j)
                r[i][q][j] = silu(__uint_as_float(v[q][j])) * __uint_as_float(up[q][j]);
            }
          }
          if (last) hand_back();
          float(*amax)[kBatch * 16] = ctl->amax[wg];
#pragma unroll
          for (int i = 0; i < kBatch; ++i) {
            if (g0 + 2 * i >= groups) break;
            float m[4];  // tokens {0, 1} and {8, 9} + 2 * (lane % 4)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int j = 4 * (q >> 1) + (q & 1);
              m[q] = fmaxf(fmaxf(fabsf(r[i][0][j]), fabsf(r[i][0][j + 2])),
                           fmaxf(fabsf(r[i][1][j]), fabsf(r[i][1][j + 2])));
#pragma unroll
              for (int o = 4; o <= 16; o <<= 1)
                m[q] = fmaxf(m[q], __shfl_xor_sync(0xffffffffu, m[q], o));
            }
            if (lane < 4) {
              *reinterpret_cast<float2*>(&amax[ew][16 * i + 2 * lane]) = make_float2(m[0], m[1]);
              *reinterpret_cast<float2*>(&amax[ew][16 * i + 8 + 2 * lane]) = make_float2(m[2], m[3]);
            }
          }
          sync_group(wg);
          auto scale_of = [&](int token) {
            const float most = fmaxf(fmaxf(amax[0][token], amax[1][token]),
                                     fmaxf(amax[2][token], amax[3][token]));
            return pow2_not_below(fmaxf(most, 1e-4f) / 448.0f);
          };
          if (lt < 16 * kBatch) {
            const int n = (g0 + 2 * (lt >> 4)) * 16 + (lt & 15);
            if (n < live)
              g.out_scale[c.expert * g.os_stride_e +
                          static_cast<int64_t>(c.first + n) * g.os_stride_row + c.w_blk] =
                  scale_of(lt);
          }
          uint8_t* seg = ctl->seg[wg];
#pragma unroll
          for (int i = 0; i < kBatch; ++i) {
            if (g0 + 2 * i >= groups) break;
#pragma unroll
            for (int b = 0; b < 2; ++b) {
              const int t0 = 16 * i + 8 * b + 2 * (lane & 3);
              const float inv0 = 1.0f / scale_of(t0), inv1 = 1.0f / scale_of(t0 + 1);
#pragma unroll
              for (int q = 0; q < 4; ++q) {  // column 8 * q + lane / 4 of this warp's 32
                const float* v = &r[i][q >> 1][4 * b + 2 * (q & 1)];
                const uint32_t e = __nv_cvt_float2_to_fp8x2(make_float2(v[0] * inv0, v[1] * inv1),
                                                            __NV_SATFINITE, __NV_E4M3);
                uint8_t* dst = seg + t0 * kSegBytesQ + ew * 32 + 8 * q + (lane >> 2);
                dst[0] = static_cast<uint8_t>(e);
                dst[kSegBytesQ] = static_cast<uint8_t>(e >> 8);
              }
            }
          }
          sync_group(wg);
#pragma unroll
          for (int i = 0; i < kBatch; ++i) {
            const int n = (g0 + 2 * i) * 16 + (lt >> 3);
            if (n < live)
              *reinterpret_cast<int4*>(static_cast<uint8_t*>(g.out) + c.expert * g.out_stride_e +
                                       static_cast<int64_t>(c.first + n) * g.out_stride_row +
                                       c.w_blk * 128 + (lt & 7) * 16) =
                  *reinterpret_cast<const int4*>(seg + (16 * i + (lt >> 3)) * kSegBytesQ +
                                                 (lt & 7) * 16);
          }
        } else {
          uint32_t v[kBatch][2][2][8];
#pragma unroll
          for (int i = 0; i < kBatch; ++i) {
            if (g0 + 2 * i >= groups) break;
            load_group(t_acc + (g0 + 2 * i) * 16, v[i][0][0], v[i][0][1]);
            load_group(t_acc + half_cols + (g0 + 2 * i) * 16, v[i][1][0], v[i][1][1]);
          }
          tc::tmem_ld_wait();
          if (last) hand_back();
#pragma unroll
          for (int ih = 0; ih < 2 * kBatch; ++ih, alt ^= 1) {
            const int grp = g0 + (ih & ~1), h = ih & 1;
            if (grp >= groups) break;
            const uint32_t(&lo)[8] = v[ih >> 1][h][0];
            const uint32_t(&hi)[8] = v[ih >> 1][h][1];
            uint8_t* seg = ctl->seg[wg] + alt * 16 * kSegBytes;
#pragma unroll
            for (int b = 0; b < 2; ++b)
              stmatrix_x4_trans(seg + (8 * b + (lane & 7)) * kSegBytes + (ew * 32 + (lane >> 3) * 8) * 2,
                                bf16_bits(lo[4 * b], lo[4 * b + 1]),
                                bf16_bits(lo[4 * b + 2], lo[4 * b + 3]),
                                bf16_bits(hi[4 * b], hi[4 * b + 1]),
                                bf16_bits(hi[4 * b + 2], hi[4 * b + 3]));
            sync_group(wg);
            const int col = c.w_blk * 256 + h * 128 + (lt & 15) * 8;
#pragma unroll
            for (int it = 0; it < 2; ++it) {
              const int tok16 = it * 8 + (lt >> 4);
              const int n = grp * 16 + tok16;
              const int4 row = *reinterpret_cast<const int4*>(seg + tok16 * kSegBytes + (lt & 15) * 16);
              if (col + 8 > g.n_out) continue;
              if constexpr (kToPeers) {
                if (peer_stage->token[n] != kNoSignal) {
                  const uint32_t first_rank = peer_stage->group[n];
                  const size_t off = peer_stage->row_off[n] + static_cast<size_t>(col) * 2;
                  for (int r = 0; r < min(p.dp_size, 8); ++r)
                    ptx::st_v4(p.peer[first_rank + r] + off, row);
                }
              } else if (n < live) {
                *reinterpret_cast<int4*>(static_cast<__nv_bfloat16*>(g.out) +
                                         c.expert * g.out_stride_e +
                                         static_cast<int64_t>(c.first + n) * g.out_stride_row + col) =
                    row;
              }
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
          const uint32_t units = static_cast<uint32_t>(min(kCols, g.n_out - c.w_blk * kCols));
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

}  // namespace mx
}  // namespace
}  // namespace pplx
