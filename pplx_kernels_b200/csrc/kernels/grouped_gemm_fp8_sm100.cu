// Block-scaled fp8 grouped expert GEMM for sm_100a (tcgen05 kind::f8f6f4).
//
//   out[e, r, :] = act( sum_kb  sa[e, r, kb] * sw[e, n / 128, kb] *
//                               (xq[e, r, kb-th 128 columns] . wq[e, n, kb-th 128 columns]) )
//
// xq / wq are e4m3, sa is one fp32 scale per row and 128 columns of K (what
// `dispatch_quant` delivers), sw one fp32 scale per 128 x 128 block of the weight
// (the DeepSeek-V3 / Qwen3 fp8 checkpoint format).  The reference has no GEMM;
// this kernel is the fp8 arm of the MoE layer that goes beyond it.
//
// Two kernels: grouped_gemm_fp8_fold.inl for arbitrary fp32 scales, which the CUDA cores apply per
// 128-wide K block, and grouped_gemm_fp8_mx.inl for power-of-two scales (`pow2_scales`), which the
// tensor cores apply.  In both the weights are the M operand and the tokens the N operand; the first
// has a form of the down projection for many rows per expert, grouped_gemm_fp8_rows.inl, with the
// tokens as the M operand.
//
// Epilogues:  plain   down projection, bf16 result
//             kSwiGLUQuant   w stacks gate and up rows; the tile is 128 gate + 128 up
//                     rows, the result silu(gate) * up is 128 columns = exactly one
//                     scale block, so it is quantised right here to e4m3 + one
//                     scale per row and tile -- the input format of the next GEMM.
//
// kFromStaging: the tokens and their scales are read out of the dispatch staging arena that
// peers fill (packed, quantising send); tiles wait for the sources they cover.
// kToPeers: the bf16 result rows go to the combine staging of the tokens' home ranks.
//
// All waits are bounded; on expiry the CTA drains, frees its tensor memory and reports through
// *status.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
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

constexpr int kBlockM = 128;
constexpr int kBlockKBytes = 128;  // 128 e4m3 values = one swizzle row = one scale block
constexpr int kUmmaKBytes = 32;
constexpr int kThreads = 384;
constexpr int kTmemCols = 512;
constexpr int kPeerTokens = 256;   // at least the widest token tile
constexpr uint32_t kWaitLimitNs = 2000000000u;
constexpr int kMaxExperts = 1024;

__device__ __forceinline__ float silu(float v) { return v / (1.0f + __expf(-v)); }

struct Fp8GemmArgs {
  const int32_t* counts;   // [E]
  const float* sa;         // [E][rows][kblocks]
  int64_t sa_stride_e, sa_stride_row;
  const float* sw;         // [E][ceil(w_rows / 128)][kblocks]
  int64_t sw_stride_e, sw_stride_row;
  void* out;               // bf16 [E][rows][n_out]  or  e4m3 [E][rows][n_out]
  int64_t out_stride_e, out_stride_row;  // elements
  float* out_scale;        // kSwiGLUQuant: [E][rows][n_out / 128]
  int64_t os_stride_e, os_stride_row;
  uint32_t* status;
  int num_experts, rows_per_expert, n_out, k;
  // Only read by the forms fused with the all-to-all:
  int32_t* out_num_tokens;  // optional [nle]: per-expert totals for the caller
  int src_table;            // keep rows per (expert, source) in shared memory
  uint32_t ring_bytes;      // shared memory for the stages (set by the launcher)
  A2AParams a2a;
};

}  // namespace
}  // namespace pplx

#include "grouped_gemm_fp8_rows.inl"
#include "grouped_gemm_fp8_fold.inl"
#include "grouped_gemm_fp8_mx.inl"

namespace pplx {
namespace {

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                   const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fp8() {
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

// [experts, rows, k] one-byte elements with k contiguous; tiles of 128 B x 128 rows x 1,
// 128-byte swizzle, out-of-range elements read as zero.
CUtensorMap make_byte_map(const void* base, int64_t experts, int64_t rows, int64_t k,
                          int64_t stride_row, int64_t stride_expert, int box_rows = 128) {
  PPLX_CHECK(reinterpret_cast<uintptr_t>(base) % 16 == 0 && stride_row % 16 == 0 &&
                 stride_expert % 16 == 0,
             "fp8 operands must be 16-byte aligned with strides that are multiples of 16");
  CUtensorMap map;
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(k), static_cast<cuuint64_t>(rows),
                              static_cast<cuuint64_t>(experts)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(stride_row),
                                 static_cast<cuuint64_t>(stride_expert)};
  const cuuint32_t box[3] = {kBlockKBytes, static_cast<cuuint32_t>(box_rows), 1};
  const cuuint32_t elem_strides[3] = {1, 1, 1};
  const CUresult r = encode_tiled_fp8()(
      &map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box,
      elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  PPLX_CHECK(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed with code " << static_cast<int>(r));
  return map;
}

}  // namespace

namespace {

constexpr size_t kMaxSrcEntriesFp8 = 2048;

void check_fp8_call(const Fp8GemmCall& c, bool need_x, bool need_out) {
  PPLX_CHECK(c.num_experts > 0 && c.num_experts <= kMaxExperts, "num_experts out of range");
  PPLX_CHECK(c.k > 0 && c.k % 16 == 0, "K must be a positive multiple of 16");
  PPLX_CHECK(c.n_out > 0 && c.n_out % 16 == 0, "the output width must be a multiple of 16");
  PPLX_CHECK(!c.swiglu_quant || c.n_out % 128 == 0,
             "the SwiGLU + quantise epilogue needs an intermediate size that is a multiple of 128");
  PPLX_CHECK(c.w && c.sw, "missing weight tensor");
  PPLX_CHECK(!need_x || (c.x && c.sa && c.counts), "missing activation tensor");
  PPLX_CHECK(!need_out || c.out, "missing output tensor");
  PPLX_CHECK(!c.swiglu_quant || c.out_scale != nullptr, "out_scale is required");
  PPLX_CHECK(reinterpret_cast<uintptr_t>(c.out) % 16 == 0, "the output must be 16-byte aligned");
}

Fp8GemmArgs fp8_args(const Fp8GemmCall& c) {
  Fp8GemmArgs g{};
  g.counts = c.counts;
  g.sa = c.sa;
  g.sa_stride_e = c.sa_stride_e;
  g.sa_stride_row = c.sa_stride_row;
  g.sw = c.sw;
  g.sw_stride_e = c.sw_stride_e;
  g.sw_stride_row = c.sw_stride_row;
  g.out = c.out;
  g.out_stride_e = c.out_stride_e;
  g.out_stride_row = c.out_stride_row;
  g.out_scale = c.out_scale;
  g.os_stride_e = c.os_stride_e;
  g.os_stride_row = c.os_stride_row;
  g.status = c.status;
  g.num_experts = c.num_experts;
  g.rows_per_expert = c.rows_per_expert;
  g.n_out = c.n_out;
  g.k = c.k;
  return g;
}

// Token rows come in boxes of 64 and 16.
struct TokenMaps {
  CUtensorMap x64, x16;
};

TokenMaps make_token_maps(const void* base, int64_t planes, int64_t rows, int64_t k,
                          int64_t stride_row, int64_t stride_plane) {
  return {make_byte_map(base, planes, rows, k, stride_row, stride_plane, 64),
          make_byte_map(base, planes, rows, k, stride_row, stride_plane, 16)};
}

// `kPow2`: the form whose scales the tensor cores apply.  `kMany`: the form for many rows per expert.
template <bool kSwiGLUQuant, bool kFromStaging, bool kToPeers, bool kPow2, bool kMany = false>
void launch_form(const CUtensorMap& tmap_w, const TokenMaps& x, Fp8GemmArgs g, int num_sms,
                 cudaStream_t stream) {
  using Control = std::conditional_t<kPow2, mx::Control, fold::Control>;
  const void* kernel;
  if constexpr (kPow2)
    kernel = reinterpret_cast<const void*>(
        &mx::grouped_gemm_fp8_mx_kernel<kSwiGLUQuant, kFromStaging, kToPeers>);
  else
    kernel = reinterpret_cast<const void*>(
        &fold::grouped_gemm_fp8_fold_kernel<kSwiGLUQuant, kFromStaging, kToPeers, kMany>);
  const size_t src_entries =
      (kFromStaging && g.src_table != 0) ? static_cast<size_t>(g.num_experts) * g.a2a.world : 0;
  const size_t fixed = 1024 + sizeof(Control) + (kToPeers ? sizeof(tok::PeerStage<kPeerTokens>) : 0) +
                       sizeof(uint32_t) * (3 * static_cast<size_t>(g.num_experts) + 1 + src_entries);
  // The stages take what the tables leave: at least two of the widest tiles beside any table the
  // checks admit, three beside those of 256 experts.
  constexpr size_t kSmem = 227 * 1024;
  static_assert(kSmem - (1024 + sizeof(Control) + sizeof(tok::PeerStage<kPeerTokens>) +
                         sizeof(uint32_t) * (3 * kMaxExperts + 1 + kMaxSrcEntriesFp8)) >=
                    2 * (mx::kWBytes + mx::kMaxTokens * kBlockKBytes) + 1024,
                "too little shared memory for the stages");
  g.ring_bytes = static_cast<uint32_t>((kSmem - fixed) & ~static_cast<size_t>(1023));
  if constexpr (kMany) {
    // (Beside the tables of several hundred experts there is no room for its stages.)
    if (g.ring_bytes < rows::kStages * rows::kStageBytes)
      return launch_form<kSwiGLUQuant, kFromStaging, kToPeers, kPow2>(tmap_w, x, g, num_sms, stream);
  }
  const size_t smem = fixed + g.ring_bytes;
  CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(smem)));
  const int grid = num_sms > 0 ? num_sms : get_sm_count();
  void* params[] = {const_cast<CUtensorMap*>(&tmap_w), const_cast<CUtensorMap*>(&x.x64),
                    const_cast<CUtensorMap*>(&x.x16), &g};
  CUDA_CHECK(launch_after_previous(kernel, dim3(grid), dim3(kThreads), params, smem, stream));
}

// Down projection with fp32 scales: whether the form for many rows needs less time, from the rows that
// the caller expects: waves of its tiles against waves of the other form's, with experts a standard
// deviation apart.  Per K block a tile of the other form takes 0.62 of what this one's, of twice the
// area, takes, in proportion to the token tile; beside their K blocks this one's epilogue is worth four
// more, and the other's four where it stores to peers.  Fitted to 124 GEMMs of seven shapes with 4 to
// 8000 rows per expert, even and skewed (mean loss against the better form 0.5 %), the last figure to
// fused layers.  E.g. 4 experts of 7168 x 2048: 100 rows each 26 us (this form 42), 4000 rows 309 (274).
bool want_many(const Fp8GemmCall& c, bool to_peers) {
  if (c.expected_total_rows <= 0) return false;
  const int grid = c.num_sms > 0 ? c.num_sms : get_sm_count();
  const double mean = std::min(static_cast<double>(c.expected_total_rows) / c.num_experts,
                               static_cast<double>(c.rows_per_expert));
  constexpr int kMost = fold::Shape<1>::kMaxTokens;
  double blocks = 0, tiles = 0;
  int width = 16;
  for (int d = -1; d <= 1; ++d) {
    const int rows = static_cast<int>(mean + d * std::sqrt(mean) + 0.5);
    if (rows <= 0) continue;
    const int t = ceil_div(rows, kMost);
    blocks += ceil_div(rows, kBlockM) / 3.0;
    tiles += t / 3.0;
    width = std::max(width, round_up(ceil_div(rows, t), 16));
  }
  auto waves = [&](double per_expert, int columns) {
    return std::max(1.0, std::ceil(per_expert * c.num_experts * ceil_div(c.n_out, columns) / grid));
  };
  const double kb = ceil_div(c.k, kBlockKBytes);
  const double here = waves(tiles, 128) * (0.62 * width / kMost * kb + (to_peers ? 4 : 0));
  return waves(blocks, rows::kTileN) * (kb + 4) < here;
}

template <bool kSwiGLUQuant, bool kFromStaging, bool kToPeers>
void launch_fp8(const Fp8GemmCall& c, const TokenMaps& x, const Fp8GemmArgs& g, cudaStream_t stream) {
  const int64_t w_rows = (kSwiGLUQuant ? 2 : 1) * static_cast<int64_t>(c.n_out);
  const CUtensorMap tmap_w =
      make_byte_map(c.w, c.num_experts, w_rows, c.k, c.w_stride_row, c.w_stride_e);
  if (c.pow2_scales)
    return launch_form<kSwiGLUQuant, kFromStaging, kToPeers, true>(tmap_w, x, g, c.num_sms, stream);
  if constexpr (!kSwiGLUQuant) {
    if (want_many(c, kToPeers))
      return launch_form<false, false, kToPeers, false, true>(tmap_w, x, g, c.num_sms, stream);
  }
  launch_form<kSwiGLUQuant, kFromStaging, kToPeers, false>(tmap_w, x, g, c.num_sms, stream);
}

}  // namespace

void launch_grouped_gemm_fp8(const Fp8GemmCall& c, cudaStream_t stream) {
  check_fp8_call(c, true, true);
  const TokenMaps x = make_token_maps(c.x, c.num_experts, c.rows_per_expert, c.k, c.x_stride_row,
                                      c.x_stride_e);
  if (c.swiglu_quant) launch_fp8<true, false, false>(c, x, fp8_args(c), stream);
  else launch_fp8<false, false, false>(c, x, fp8_args(c), stream);
}

void launch_gemm_fp8_from_staging(const Fp8GemmCall& c, const A2AParams& p,
                                  int32_t* out_num_tokens, cudaStream_t stream) {
  check_fp8_call(c, false, true);
  PPLX_CHECK(c.swiglu_quant, "the staging-fed fp8 GEMM is the SwiGLU up projection");
  PPLX_CHECK(p.hidden_bytes == p.hidden_dim && p.scale_bytes == ceil_div(p.hidden_dim, 128) * 4,
             "the staging-fed fp8 GEMM needs an object created for a 1-byte payload with one "
             "fp32 scale per 128 columns");
  PPLX_CHECK(c.k == p.hidden_dim && c.num_experts == p.nle && c.rows_per_expert >= p.cap,
             "shape mismatch between the GEMM and the all-to-all");
  // Tokens: [1][world * region_slots][hidden] e4m3 view of this rank's packed staging.
  const int64_t slots = static_cast<int64_t>(p.world) * p.region_slots;
  const TokenMaps x = make_token_maps(p.peer[p.rank] + p.off_disp_stage, 1, slots, p.hidden_dim,
                                      p.slot_bytes, slots * p.slot_bytes);
  Fp8GemmArgs g = fp8_args(c);
  g.out_num_tokens = out_num_tokens;
  g.a2a = p;
  g.src_table = static_cast<size_t>(p.nle) * p.world <= kMaxSrcEntriesFp8 ? 1 : 0;
  launch_fp8<true, true, false>(c, x, g, stream);
}

void launch_gemm_fp8_to_peers(const Fp8GemmCall& c, const A2AParams& p, cudaStream_t stream) {
  check_fp8_call(c, true, false);
  PPLX_CHECK(!c.swiglu_quant, "the peer-storing fp8 GEMM is the plain down projection");
  PPLX_CHECK(c.n_out == p.hidden_dim && c.num_experts == p.nle && c.rows_per_expert >= p.cap,
             "shape mismatch between the GEMM and the all-to-all");
  PPLX_CHECK(c.counts == reinterpret_cast<const int32_t*>(p.recv_count),
             "counts must be the all-to-all's received-row counts");
  PPLX_CHECK(p.dp_size <= 8, "at most 8 replicas per DP group");
  const TokenMaps x = make_token_maps(c.x, c.num_experts, c.rows_per_expert, c.k, c.x_stride_row,
                                      c.x_stride_e);
  Fp8GemmArgs g = fp8_args(c);
  g.out = nullptr;
  g.a2a = p;
  launch_fp8<false, false, true>(c, x, g, stream);
}

}  // namespace pplx
