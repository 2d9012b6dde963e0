// What the steps of the grouped (per-expert) path share inside the library.
#pragma once

#include "common.cuh"

namespace b200fp4 {

constexpr int kGroupMaxExperts = 4096;
constexpr int kGroupTileRows = 128;            // rows of a grouped-GEMM tile

// The tile list of the grouped GEMM, at the start of its workspace: status word (0 = ok) | ... | hdr (int 4): number of tiles |
// ... | (byte 256) per tile {first row, end row of its expert, scale-tile row of A, expert}.
inline int* grouped_status(void* ws) { return static_cast<int*>(ws); }
inline int* grouped_hdr(void* ws) { return static_cast<int*>(ws) + 4; }
inline int4* grouped_tiles(void* ws) { return reinterpret_cast<int4*>(static_cast<unsigned char*>(ws) + 256); }
inline int grouped_max_tiles(int64_t rows, int64_t E) { return (int)(rows / kGroupTileRows + E + 1); }

// Routing metadata; with tile_ws also the tile list.  At most kRouteMaxPairs pairs.  dst2src may be null.  (moe_prefill.cu)
constexpr int64_t kRouteMaxPairs = 131072;
void launch_moe_route(const int32_t* topk_ids, int P, const int32_t* expert_map, int global_E, int E, int32_t* expert_offsets,
                      int32_t* blockscale_offsets, int32_t* dst2src, int32_t* src2dst, void* tile_ws, cudaStream_t st);

// Token-major quantization (b200fp4_experts_quantize_scatter).  stage_sf: the block scales go to the layout that only the
// grouped GEMM reads, [128-row tile][256 of k][row][16 bytes] (K % 64 == 0; stage_sf_bytes()): a stage of the GEMM is 2 KB in a
// piece as in the swizzled layout, but a row's scales are stored 16 bytes at a time instead of 4.  The scale bytes of padding
// rows then stay undefined, which the grouped GEMM does not mind: they only scale rows that are never stored.  (quant.cu)
inline size_t stage_sf_bytes(int64_t padded_rows, int64_t K) { return (size_t)padded_rows * (size_t)((K + 255) / 256 * 16); }
int experts_quantize_scatter(const void* x, int in_dtype, int64_t n_src, int64_t K, int64_t topk, const int32_t* src2dst,
                             const float* global_scales, const int32_t* expert_offsets, const int32_t* blockscale_offsets,
                             int32_t num_experts, int64_t sf_rows_padded, const int32_t* topk_ids, const int32_t* expert_map,
                             int64_t global_E, void* codes, void* sf, void* stream, bool stage_sf);
// What it refuses, without queueing anything.
int experts_quantize_scatter_check(const void* x, int in_dtype, int64_t n_src, int64_t K, int64_t topk, const int32_t* src2dst,
                                   const float* global_scales, const int32_t* expert_offsets, const int32_t* blockscale_offsets,
                                   int32_t num_experts, int64_t sf_rows_padded, const int32_t* topk_ids, const int32_t* expert_map,
                                   int64_t global_E, const void* codes, const void* sf, bool stage_sf);

// The grouped GEMM; q_sf / q_gs non-null: the gate_up projection with SiLU(gate)*up and the NVFP4 quantization of the result
// in the epilogue (out = packed codes [rows_capacity, N/4]).  tiles_ready: the workspace already holds the tile list.  stage_sf:
// a_sf is in the layout above (gate_up only).  (gemm.cu)
int grouped_gemm(const void* a_codes, const void* b_codes, const void* a_sf, const void* b_sf, const float* alphas,
                 const int32_t* expert_offsets, const int32_t* sf_offsets, void* out, int out_dtype, int64_t rows_capacity, int64_t N,
                 int64_t K, int64_t E, int tile_n, void* workspace, size_t workspace_bytes, void* stream, void* q_sf, const float* q_gs,
                 bool tiles_ready, bool stage_sf);
// What it refuses of its arguments, without queueing anything (the device is not looked at).
int grouped_gemm_check(const void* a_codes, const void* b_codes, const void* a_sf, const void* b_sf, const float* alphas,
                       const int32_t* expert_offsets, const int32_t* sf_offsets, const void* out, int out_dtype, int64_t rows_capacity,
                       int64_t N, int64_t K, int64_t E, int tile_n, const void* workspace, size_t workspace_bytes, const void* q_sf,
                       const float* q_gs, bool stage_sf);

}  // namespace b200fp4
