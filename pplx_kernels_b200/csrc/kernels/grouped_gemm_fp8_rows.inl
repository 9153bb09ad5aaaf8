// fp8 expert GEMM with fp32 scales, the down projection's form for many rows per expert (included by
// grouped_gemm_fp8_sm100.cu): the TOKENS are the M operand, a tile is 128 of them times 256 weight
// rows.
//
// The form with the tokens as N (grouped_gemm_fp8_fold.inl) follows the rows there are, which is what
// counts up to about a hundred per expert.  Beyond, its plain tiles of 128 weight rows are half of
// these: an MMA reads its 128 weight rows from shared memory for 128 columns instead of 256, and
// the peer-storing epilogue announces every row twice as often (an add per row and tile, over NVLink).
// The SwiGLU form and the kernel for power-of-two scales have nothing like it: there the form with the
// tokens as N is level or ahead at every size.
//
// Layers in fp8 with the other form / this one for the down projection: 32 DeepSeek-V3 experts,
// fused, 800 tokens 625 / 579 us, 2048 tokens 1343 / 1209; DeepSeek-V2-Lite, fused, 4096 tokens
// 550 / 503; Mixtral 8x7B, 2048 tokens 1200 / 1154, with 512 tokens 394 / 424.
//
// Every 128-wide K block is multiplied into one of two scratch accumulators and folded, times the two
// scales, into 128 sums per thread by eight warps; a thread owns a row and half of its columns.  Roles:
// warp 0 TMA producer, warp 1 MMA issuer, warps 4-11 fold and epilogue.
namespace pplx {
namespace {
namespace rows {

constexpr int kTileN = 256;  // weight rows per tile
constexpr uint32_t kABytes = kBlockM * kBlockKBytes;
constexpr uint32_t kBBytes = kTileN * kBlockKBytes;
constexpr uint32_t kStageBytes = kABytes + kBBytes;
constexpr uint32_t kStages = 4;  // (as a number that the launch decides it cost up to 5 %)
// Peer-storing epilogue: 64 bytes of a row pass through shared memory at a time, as four pieces of
// 16 bytes that change places from one pair of rows to the next (bank conflicts).
constexpr int kRowPieceBytes = 64;
constexpr uint32_t kScratchBytes = 8 * 32 * kRowPieceBytes;
__device__ __forceinline__ int piece_at(int row, int piece) {
  return (piece ^ ((row >> 1) & 3)) * 16;
}

struct Barriers {
  uint64_t full[kStages];
  uint64_t empty[kStages];
  uint64_t part_full[2];   // scratch accumulator holds a finished K block
  uint64_t part_empty[2];  // ... may be overwritten
};

__device__ __forceinline__ void init_barriers(Barriers* bar) {
  for (uint32_t s = 0; s < kStages; ++s) {
    tc::mbar_init(&bar->full[s], 1);
    tc::mbar_init(&bar->empty[s], 1);
  }
  for (int b = 0; b < 2; ++b) {
    tc::mbar_init(&bar->part_full[b], 1);
    tc::mbar_init(&bar->part_empty[b], 8);
  }
}

struct Tile {
  int expert, m_blk, n_blk, rows;
};

__device__ __forceinline__ Tile locate(const uint32_t* tile_start, const uint32_t* rows_of,
                                       int num_experts, uint32_t t) {
  Tile c;
  c.expert = find_group(tile_start, num_experts, t);
  c.rows = static_cast<int>(rows_of[c.expert]);
  const int m_tiles = ceil_div<int>(c.rows, kBlockM);
  const uint32_t rem = t - tile_start[c.expert];
  c.n_blk = static_cast<int>(rem / m_tiles);
  c.m_blk = static_cast<int>(rem - static_cast<uint32_t>(c.n_blk) * m_tiles);
  return c;
}

// What the kernel around this form has set up.
struct Shared {
  uint8_t* ring;            // shared memory of the stages
  Barriers* bar;
  uint8_t* scratch;         // kScratchBytes
  tok::PeerStage<kPeerTokens>* peer_stage;
  uint32_t* tile_start;     // [E + 1]; rewritten
  const uint32_t* rows_of;  // [E]
  volatile uint32_t* abort_flag;
  uint32_t tmem_base;
};

// 32 lanes x 16 consecutive columns.
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}

__device__ __forceinline__ int4 pack8_bf16(const float* v) {
  int4 o;
  uint32_t* w = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
    w[j] = *reinterpret_cast<const uint32_t*>(&b);
  }
  return o;
}

// All threads of the block.  Returns with all roles of the calling warp done.
template <bool kToPeers>
__device__ __forceinline__ void run(const CUtensorMap& tmap_w, const CUtensorMap& tmap_x64,
                                    const Fp8GemmArgs& g, const Shared& x) {
  const A2AParams& p = g.a2a;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n_blocks = ceil_div<int>(g.n_out, kTileN);
  const int num_kb = ceil_div<int>(g.k, kBlockKBytes);
  auto* peer_stage = x.peer_stage;
  __syncthreads();  // everybody has read the tables of the other form
  for (int e = tid; e < g.num_experts; e += blockDim.x)
    x.tile_start[e] =
        static_cast<uint32_t>(ceil_div<int>(static_cast<int>(x.rows_of[e]), kBlockM) * n_blocks);
  __syncthreads();
  if (warp == 0) warp_exclusive_scan_smem(x.tile_start, g.num_experts, lane, true);
  __syncthreads();
  const uint32_t total_tiles = x.tile_start[g.num_experts];

  if (warp == 0) {
    if (tc::elect_one()) {
      uint32_t stage = 0, phase = 0, pending = 0, pending_phase = 0;
      bool ok = *x.abort_flag == 0u;
      for (uint32_t t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
        const Tile c = locate(x.tile_start, x.rows_of, g.num_experts, t);
        const int a_row = c.m_blk * kBlockM;
        // Of a last block with 64 rows at most, only the first half is fetched: the results of the
        // other rows are not stored.
        const bool both = c.rows - a_row > kBlockM / 2;
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = tc::mbar_wait(&x.bar->empty[stage], phase ^ 1u, x.abort_flag, kWaitLimitNs);
          if (!ok) break;
          uint8_t* a_dst = x.ring + stage * kStageBytes;
          uint8_t* b_dst = a_dst + kABytes;
          uint64_t* full = &x.bar->full[stage];
          tc::mbar_arrive_expect_tx(full, kStageBytes - (both ? 0u : kABytes / 2));
          pending |= 1u << stage;
          pending_phase = (pending_phase & ~(1u << stage)) | (phase << stage);
          const int k0 = kb * kBlockKBytes;
          tc::tma_load_3d(a_dst, &tmap_x64, full, k0, a_row, c.expert);
          if (both)
            tc::tma_load_3d(a_dst + kABytes / 2, &tmap_x64, full, k0, a_row + kBlockM / 2, c.expert);
          tc::tma_load_3d(b_dst, &tmap_w, full, k0, c.n_blk * kTileN, c.expert);
          tc::tma_load_3d(b_dst + kBBytes / 2, &tmap_w, full, k0, c.n_blk * kTileN + kTileN / 2,
                          c.expert);
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      if (!ok || *x.abort_flag != 0u) {
        const uint64_t t0 = ptx::globaltimer_ns();
        for (uint32_t s = 0; s < kStages; ++s) {
          if (!((pending >> s) & 1u)) continue;
          while (!tc::mbar_try_wait(&x.bar->full[s], (pending_phase >> s) & 1u)) {
            if (ptx::globaltimer_ns() - t0 > 100000000ull) break;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (tc::elect_one()) {
      // kind::f8f6f4, e4m3 x e4m3 -> f32, M = 128, N = 256.
      const uint32_t idesc = tc::make_instr_desc(0u, kBlockM, kTileN);
      uint32_t stage = 0, phase = 0, round = 0;
      bool ok = *x.abort_flag == 0u;
      for (uint32_t t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
        for (int kb = 0; kb < num_kb && ok; ++kb, ++round) {
          // K blocks alternate between the two scratch accumulators.
          const uint32_t buf = round & 1u;
          ok = tc::mbar_wait(&x.bar->part_empty[buf], ((round >> 1) & 1u) ^ 1u, x.abort_flag,
                             kWaitLimitNs) &&
               tc::mbar_wait(&x.bar->full[stage], phase, x.abort_flag, kWaitLimitNs);
          if (!ok) break;
          tc::tc_fence_after_sync();
          const uint8_t* a_src = x.ring + stage * kStageBytes;
          const uint64_t a_desc = tc::make_smem_desc_sw128(a_src);
          const uint64_t b_desc = tc::make_smem_desc_sw128(a_src + kABytes);
#pragma unroll
          for (int k = 0; k < kBlockKBytes / kUmmaKBytes; ++k) {
            tc::mma_f8_ss(x.tmem_base + buf * kTileN, tc::advance_smem_desc(a_desc, k * kUmmaKBytes),
                          tc::advance_smem_desc(b_desc, k * kUmmaKBytes), idesc, k != 0);
          }
          tc::mma_commit(&x.bar->empty[stage]);
          tc::mma_commit(&x.bar->part_full[buf]);
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp >= 4) {
    const int ew = (warp - 4) & 3;     // tensor-memory lanes [32 * ew, +32)
    const int half = (warp - 4) >> 2;  // columns [64 * half, +64) of each 128-column half
    const uint32_t t_lane = x.tmem_base + (static_cast<uint32_t>(ew * 32) << 16);
    uint32_t round = 0;
    uint32_t pending_signals = 0;  // kToPeers, warp 4: queued arrival adds
    bool ok = *x.abort_flag == 0u;
    for (uint32_t t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
      const Tile c = locate(x.tile_start, x.rows_of, g.num_experts, t);
      const int tile_row = ew * 32 + lane;
      const int row = c.m_blk * kBlockM + tile_row;
      const bool row_ok = row < c.rows;
      const float* sa_row = g.sa + c.expert * g.sa_stride_e + (row_ok ? row : 0) * g.sa_stride_row;
      // Weight scale rows of the two halves of the tile.
      const int last_block = (g.n_out - 1) / 128;
      const float* sw0 =
          g.sw + c.expert * g.sw_stride_e + min(2 * c.n_blk, last_block) * g.sw_stride_row;
      const float* sw1 =
          g.sw + c.expert * g.sw_stride_e + min(2 * c.n_blk + 1, last_block) * g.sw_stride_row;

      // acc[0..63]: columns 64*half.. of the first 128-column half of the tile,
      // acc[64..127]: the same columns of the second half.
      float acc[128];
#pragma unroll
      for (int j = 0; j < 128; ++j) acc[j] = 0.f;
      for (int kb = 0; kb < num_kb && ok; ++kb, ++round) {
        const float a_scale = __ldg(sa_row + kb);
        const float s0 = a_scale * __ldg(sw0 + kb);
        const float s1 = a_scale * __ldg(sw1 + kb);
        const uint32_t buf = round & 1u;
        ok = tc::mbar_wait(&x.bar->part_full[buf], (round >> 1) & 1u, x.abort_flag, kWaitLimitNs);
        if (!ok) break;
        tc::tc_fence_after_sync();
        const uint32_t t_part = t_lane + buf * kTileN + half * 64;
#pragma unroll
        for (int q = 0; q < 8; ++q) {  // 8 pieces of 16 columns: 4 per tile half
          uint32_t part[16];
          tmem_ld_32x16(t_part + (q >> 2) * 128 + (q & 3) * 16, part);
          tc::tmem_ld_wait();
          const float s = (q >> 2) == 0 ? s0 : s1;
#pragma unroll
          for (int j = 0; j < 16; ++j)
            acc[q * 16 + j] = fmaf(__uint_as_float(part[j]), s, acc[q * 16 + j]);
        }
        tc::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&x.bar->part_empty[buf]);
      }
      // All eight epilogue warps leave together or not at all: the barriers below must
      // never be entered by only some of them.
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

      // ---- tile epilogue ------------------------------------------------------
      if constexpr (kToPeers) {
        // Where each row goes, and whose token it is.  Looked up only now, so that the pointers are
        // not live across the K loop.
        if (half == 0) {
          unsigned long long off = 0;
          uint32_t sig_token = tok::kNoSignal, sig_group = 0;
          if (row_ok) {
            const uint2 rs = p.row_src[static_cast<size_t>(c.expert) * p.cap + row];
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
          peer_stage->token[tile_row] = sig_token;
          peer_stage->group[tile_row] = sig_group;
          peer_stage->row_off[tile_row] = off;
        }
        asm volatile("bar.sync 2, 256;" ::: "memory");
        // A thread owns one row; stored straight from registers its 16-byte pieces would cross
        // NVLink one by one.  Each warp passes 32 columns at a time through shared memory and writes
        // them out as 64-byte row segments (four lanes per row).
        const int replicas = min(p.dp_size, 8);
        uint8_t* stg = x.scratch + (warp - 4) * 32 * kRowPieceBytes;
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {  // 32 columns of this thread's 128
#pragma unroll
          for (int v4 = 0; v4 < 4; ++v4)
            *reinterpret_cast<int4*>(stg + lane * kRowPieceBytes + piece_at(lane, v4)) =
                pack8_bf16(acc + (q4 * 4 + v4) * 8);
          __syncwarp();
          const int seg = lane & 3;
          const int col = c.n_blk * kTileN + (q4 >> 1) * 128 + half * 64 + (q4 & 1) * 32 + seg * 8;
#pragma unroll 2
          for (int it = 0; it < 4; ++it) {
            const int rr = it * 8 + (lane >> 2);
            const int trow = ew * 32 + rr;
            if (peer_stage->token[trow] != tok::kNoSignal && col + 8 <= g.n_out) {
              const int4 o =
                  *reinterpret_cast<const int4*>(stg + rr * kRowPieceBytes + piece_at(rr, seg));
              const uint32_t grp = peer_stage->group[trow];
              const size_t off = peer_stage->row_off[trow] + static_cast<size_t>(col) * 2;
              for (int r = 0; r < replicas; ++r) ptx::st_v4(p.peer[grp + r] + off, o);
            }
          }
          __syncwarp();
        }
        // Arrival is counted in columns: this tile's share of each row.  The adds are queued and
        // flushed behind ONE system-scope fence for as many tiles as the queue holds.  (All eight
        // warps meet at the barrier at the top of the next tile's epilogue before anyone rewrites
        // the table.)
        asm volatile("bar.sync 3, 256;" ::: "memory");
        if (warp == 4) {
          const uint32_t units = static_cast<uint32_t>(min(kTileN, g.n_out - c.n_blk * kTileN));
          if (pending_signals + kBlockM > tok::kQueue) {
            tok::flush(p, peer_stage, pending_signals, lane);
            pending_signals = 0;
          }
          for (int j = lane; j < kBlockM; j += 32) {
            const uint32_t token = peer_stage->token[j];
            const bool there = token != tok::kNoSignal;
            const uint32_t mask = __ballot_sync(0xffffffffu, there);
            if (there) {
              const uint32_t at = pending_signals + __popc(mask & ((1u << lane) - 1u));
              peer_stage->q_token[at] = token;
              peer_stage->q_group_units[at] = peer_stage->group[j] | (units << 8);
            }
            pending_signals += __popc(mask);
          }
          __syncwarp();
        }
      } else if (row_ok) {
        __nv_bfloat16* orow = static_cast<__nv_bfloat16*>(g.out) + c.expert * g.out_stride_e +
                              static_cast<int64_t>(row) * g.out_stride_row;
#pragma unroll
        for (int v = 0; v < 16; ++v) {  // 16 vectors of 8 columns
          const int col = c.n_blk * kTileN + (v >> 3) * 128 + half * 64 + (v & 7) * 8;
          if (col + 8 > g.n_out) continue;
          *reinterpret_cast<int4*>(orow + col) = pack8_bf16(acc + v * 8);
        }
      }
    }
    if constexpr (kToPeers) {
      // What is still queued (also after a failed wait: rows that were stored are announced).
      if (warp == 4 && pending_signals > 0) tok::flush(p, peer_stage, pending_signals, lane);
    }
  }
}

}  // namespace rows
}  // namespace
}  // namespace pplx
