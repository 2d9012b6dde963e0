// One MoE layer over dense NVFP4 expert weights in one call: routing metadata -> token-major quantization -> grouped
// gate_up GEMM with SiLU*up and quantization in its epilogue -> grouped down GEMM -> un-permute and weighted sum (the flow of
// vllm/model_executor/layers/fused_moe/experts/cutlass_moe.py:567-663).  Issued as separate Python calls a prompt of a few
// hundred tokens spent 130 us on the host for 200 us of kernels.
#include "grouped.cuh"

namespace b200fp4 {
namespace {

// ------------------------------------------------------------------------------------------ routing metadata

// Routing metadata of up to kRouteMaxPairs pairs in one launch of one cluster of eight blocks:
//   expert_offsets[E+1]      first permuted row of every expert
//   blockscale_offsets[E+1]  the same with every expert padded to a multiple of 128 rows
//   dst2src[P]               permuted row -> pair index (token*topk + slot); -1 past the last valid row (optional)
//   src2dst[P]               pair index -> permuted row, or -1 if the pair's expert is not local
//   hdr, mtiles              the grouped GEMM's tile list (optional)
// All of it is latency: each block counts its share of the pairs per expert in shared memory (an atomic's return value is the
// pair's rank, kept in a register), the blocks add each other's counts through distributed shared memory, and every block
// scans the totals for itself.  8192 tokens, top-10, 512 experts: four grid-wide kernels and a separate tile-list kernel per
// GEMM took 24 us of kernels and six launches.
constexpr int kRouteBlocks = 8;
constexpr int kRouteThreads = 1024;
constexpr int kRoutePer = (int)(kRouteMaxPairs / (kRouteBlocks * kRouteThreads));      // pairs per thread
static_assert(kRoutePer * kRouteBlocks * kRouteThreads == kRouteMaxPairs, "pairs per thread");

__device__ __forceinline__ int cluster_load(const int* smem_here, uint32_t rank) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(smem_here), remote;
  int v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(remote) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__global__ void __cluster_dims__(kRouteBlocks, 1, 1) __launch_bounds__(kRouteThreads)
    moe_route_kernel(const int32_t* __restrict__ topk_ids, int P, const int32_t* __restrict__ expert_map, int global_E, int E,
                     int* expert_offsets, int* blockscale_offsets, int* dst2src, int* src2dst, int* hdr, int4* mtiles, int max_tiles) {
  __shared__ int s_count[kGroupMaxExperts];      // pairs of this block per expert
  __shared__ int s_first[kGroupMaxExperts];      // permuted row of this block's first pair of an expert
  __shared__ int s_warp[2][kRouteThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t rank = blockIdx.x;
  for (int e = tid; e < E; e += kRouteThreads) s_count[e] = 0;
  pdl_wait();
  pdl_launch_dependents();
  __syncthreads();
  int er[kRoutePer];                             // expert << 16 | rank among this block's pairs of it, or -1
#pragma unroll
  for (int i = 0; i < kRoutePer; ++i) {
    const int p = (i * kRouteBlocks + (int)rank) * kRouteThreads + tid;
    er[i] = p < P ? topk_ids[p] : -1;            // all in flight together
  }
#pragma unroll
  for (int i = 0; i < kRoutePer; ++i) {
    const int p = (i * kRouteBlocks + (int)rank) * kRouteThreads + tid;
    if (p < P) {
      int e = er[i];
      er[i] = -1;
      if (expert_map != nullptr) e = (e >= 0 && e < global_E) ? expert_map[e] : -1;
      if (e >= 0 && e < E) er[i] = e << 16 | atomicAdd(&s_count[e], 1);
    }
  }
  cluster_barrier();
  // every block scans the totals of all blocks; each thread owns a contiguous run of experts
  constexpr int kMaxPer = kGroupMaxExperts / kRouteThreads;
  const int per = (E + kRouteThreads - 1) / kRouteThreads;
  int total[kMaxPer], before[kMaxPer], rows = 0, tiles = 0;
#pragma unroll
  for (int i = 0; i < kMaxPer; ++i) {
    total[i] = before[i] = 0;
    const int e = tid * per + i;
    if (i < per && e < E) {
#pragma unroll
      for (uint32_t c = 0; c < kRouteBlocks; ++c) {
        const int v = cluster_load(&s_count[e], c);
        total[i] += v;
        before[i] += c < rank ? v : 0;
      }
    }
    rows += total[i];
    tiles += (total[i] + kGroupTileRows - 1) / kGroupTileRows;
  }
  int inc_r = rows, inc_t = tiles;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, inc_r, d), b = __shfl_up_sync(0xffffffffu, inc_t, d);
    if (lane >= d) {
      inc_r += a;
      inc_t += b;
    }
  }
  if (lane == 31) {
    s_warp[0][warp] = inc_r;
    s_warp[1][warp] = inc_t;
  }
  __syncthreads();
  if (warp == 0) {
    int a = s_warp[0][lane], b = s_warp[1][lane];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, a, d), y = __shfl_up_sync(0xffffffffu, b, d);
      if (lane >= d) {
        a += x;
        b += y;
      }
    }
    s_warp[0][lane] = a;
    s_warp[1][lane] = b;
  }
  __syncthreads();
  int row = inc_r - rows + (warp > 0 ? s_warp[0][warp - 1] : 0), tile = inc_t - tiles + (warp > 0 ? s_warp[1][warp - 1] : 0);
  const int all_rows = s_warp[0][31], all_tiles = s_warp[1][31];
#pragma unroll
  for (int i = 0; i < kMaxPer; ++i) {
    const int e = tid * per + i;
    if (i < per && e < E) {
      const int nt = (total[i] + kGroupTileRows - 1) / kGroupTileRows;
      s_first[e] = row + before[i];
      if (rank == 0) {
        expert_offsets[e] = row;
        blockscale_offsets[e] = tile * kGroupTileRows;
      }
      if (mtiles != nullptr)                     // the blocks share the tiles of an expert
        for (int t = (int)rank; t < nt; t += kRouteBlocks)
          if (tile + t < max_tiles) mtiles[tile + t] = make_int4(row + t * kGroupTileRows, row + total[i], tile + t, e);
      row += total[i];
      tile += nt;
    }
  }
  if (rank == 0 && tid == 0) {
    expert_offsets[E] = all_rows;
    blockscale_offsets[E] = all_tiles * kGroupTileRows;
    if (hdr != nullptr) {
      hdr[-4] = 0;                               // the GEMM's status word
      hdr[0] = min(all_tiles, max_tiles);
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kRoutePer; ++i) {
    const int p = (i * kRouteBlocks + (int)rank) * kRouteThreads + tid;
    if (p < P) {
      const int pos = er[i] < 0 ? -1 : s_first[er[i] >> 16] + (er[i] & 0xFFFF);
      src2dst[p] = pos;
      if (dst2src != nullptr) {
        if (pos >= 0) dst2src[pos] = p;
        if (p >= all_rows) dst2src[p] = -1;
      }
    }
  }
  cluster_barrier();                             // no block leaves while another may still read its counts
}

// The same routing metadata for more pairs than that, as three grid-wide steps around global counters kept in
// expert_offsets itself (no scratch): count pairs per expert, scan, scatter with expert_offsets[e] as
// the running cursor, then shift the cursors (now each expert's end) back into start offsets.
// Both grid-wide passes aggregate per block in shared memory first: with skewed routing a popular expert would
// otherwise take one global atomic per pair on a single address.
constexpr int kPermuteBlock = 1024;

__global__ void __launch_bounds__(kPermuteBlock)
    moe_permute_count_kernel(const int32_t* __restrict__ topk_ids, int P, const int32_t* __restrict__ expert_map,
                             int global_E, int E, int* expert_offsets, int* dst2src, int* src2dst) {
  __shared__ int s_count[kGroupMaxExperts];
  for (int e = threadIdx.x; e < E; e += kPermuteBlock) s_count[e] = 0;
  __syncthreads();
  const int p = blockIdx.x * kPermuteBlock + threadIdx.x;
  if (p < P) {
    int e = topk_ids[p];
    if (expert_map != nullptr) e = (e >= 0 && e < global_E) ? expert_map[e] : -1;
    if (e < 0 || e >= E) e = -1;
    src2dst[p] = e;
    dst2src[p] = -1;
    if (e >= 0) atomicAdd(&s_count[e], 1);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += kPermuteBlock) {
    const int c = s_count[e];
    if (c > 0) atomicAdd(&expert_offsets[e], c);
  }
}

__global__ void __launch_bounds__(1024)
    moe_permute_scan_kernel(int E, int* expert_offsets, int* blockscale_offsets) {
  __shared__ int s_scan[1024], s_scan2[1024];
  const int tid = threadIdx.x;
  const int per = (E + 1023) / 1024;
  int sum = 0, sum_pad = 0;
  for (int i = 0; i < per; ++i) {
    const int e = tid * per + i;
    if (e < E) {
      const int c = expert_offsets[e];
      sum += c;
      sum_pad += (c + 127) / 128 * 128;
    }
  }
  s_scan[tid] = sum;
  s_scan2[tid] = sum_pad;
  __syncthreads();
  for (int d = 1; d < 1024; d <<= 1) {
    const int v = tid >= d ? s_scan[tid - d] : 0, v2 = tid >= d ? s_scan2[tid - d] : 0;
    __syncthreads();
    s_scan[tid] += v;
    s_scan2[tid] += v2;
    __syncthreads();
  }
  int base = s_scan[tid] - sum, base_pad = s_scan2[tid] - sum_pad;
  for (int i = 0; i < per; ++i) {
    const int e = tid * per + i;
    if (e < E) {
      const int c = expert_offsets[e];
      expert_offsets[e] = base;
      blockscale_offsets[e] = base_pad;
      base += c;
      base_pad += (c + 127) / 128 * 128;
    }
  }
  if (tid == 1023) {
    expert_offsets[E] = s_scan[1023];
    blockscale_offsets[E] = s_scan2[1023];
  }
}

__global__ void __launch_bounds__(kPermuteBlock)
    moe_permute_scatter_kernel(int P, int E, int* expert_offsets, int* dst2src, int* src2dst) {
  __shared__ int s_count[kGroupMaxExperts];     // pairs of this block per expert, then the block's first row
  for (int e = threadIdx.x; e < E; e += kPermuteBlock) s_count[e] = 0;
  __syncthreads();
  const int p = blockIdx.x * kPermuteBlock + threadIdx.x;
  int e = -1, rank = 0;
  if (p < P) {
    e = src2dst[p];
    if (e >= 0) rank = atomicAdd(&s_count[e], 1);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < E; i += kPermuteBlock) {
    const int c = s_count[i];
    if (c > 0) s_count[i] = atomicAdd(&expert_offsets[i], c);
  }
  __syncthreads();
  if (e >= 0) {
    const int pos = s_count[e] + rank;
    src2dst[p] = pos;
    dst2src[pos] = p;
  }
}

__global__ void __launch_bounds__(1024) moe_permute_shift_kernel(int E, int* expert_offsets) {
  __shared__ int s_end[kGroupMaxExperts];
  for (int e = threadIdx.x; e < E; e += 1024) s_end[e] = expert_offsets[e];
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += 1024) expert_offsets[e + 1] = s_end[e];
  if (threadIdx.x == 0) expert_offsets[0] = 0;
}

// ------------------------------------------------------------------------------------------ un-permute

// out[m, h] = sum over the token's slots of weight * expert_out[src2dst[m*topk + t], h] (local pairs only).
template <typename T>
__global__ void unpermute_reduce_kernel(const T* __restrict__ expert_out, const int* __restrict__ src2dst,
                                        const float* __restrict__ topk_w, int M, int topk, int H, T* __restrict__ out) {
  const int m = blockIdx.y;
  for (int h = (blockIdx.x * blockDim.x + threadIdx.x) * 2; h < H; h += gridDim.x * blockDim.x * 2) {
    float a0 = 0.f, a1 = 0.f;
    for (int t = 0; t < topk; ++t) {
      const int r = src2dst[m * topk + t];
      if (r < 0) continue;
      const float w = topk_w[m * topk + t];
      a0 = fmaf(w, to_f32<T>(expert_out[(int64_t)r * H + h]), a0);
      a1 = fmaf(w, to_f32<T>(expert_out[(int64_t)r * H + h + 1]), a1);
    }
    out[(int64_t)m * H + h] = from_f32<T>(a0);
    out[(int64_t)m * H + h + 1] = from_f32<T>(a1);
  }
}

// The same for H % 8 == 0 and 16-byte aligned rows: eight columns per thread, 16-byte loads and stores, same order of
// additions per output element.  Bound by HBM (the rows of a large prompt do not fit L2) or, for small prompts, by the latency
// of a token's rows: those of four slots are requested before the first is used (8192 x 2048, ten slots: four 68 us, five 67.5,
// eight 73.5, twelve 84.6 -- their registers cost more warps than they keep requests in flight).
constexpr int kUnpermuteThreads = 128, kUnpermuteBatch = 4;

template <typename T>
__global__ void __launch_bounds__(kUnpermuteThreads)
    unpermute_reduce_vec8_kernel(const T* __restrict__ expert_out, const int* __restrict__ src2dst,
                                 const float* __restrict__ topk_w, int M, int topk, int H, T* __restrict__ out) {
  pdl_wait();
  pdl_launch_dependents();
  const int m = blockIdx.y;
  const int h = (blockIdx.x * kUnpermuteThreads + threadIdx.x) * 8;
  if (h >= H) return;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int t0 = 0; t0 < topk; t0 += kUnpermuteBatch) {
    uint4 raw[kUnpermuteBatch];
    float w[kUnpermuteBatch];
#pragma unroll
    for (int i = 0; i < kUnpermuteBatch; ++i) {
      const int r = t0 + i < topk ? src2dst[m * topk + t0 + i] : -1;
      raw[i] = make_uint4(0, 0, 0, 0);
      w[i] = 0.f;
      if (r >= 0) {
        raw[i] = ldg_stream_u4(expert_out + (int64_t)r * H + h);
        w[i] = topk_w[m * topk + t0 + i];
      }
    }
#pragma unroll
    for (int i = 0; i < kUnpermuteBatch; ++i) {
      const T* v = reinterpret_cast<const T*>(&raw[i]);
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] = fmaf(w[i], to_f32<T>(v[k]), acc[k]);
    }
  }
  uint4 o;
  T* ov = reinterpret_cast<T*>(&o);
#pragma unroll
  for (int i = 0; i < 8; ++i) ov[i] = from_f32<T>(acc[i]);
  *reinterpret_cast<uint4*>(out + (int64_t)m * H + h) = o;
}

// ------------------------------------------------------------------------------------------ the layer in one call

size_t part(size_t v) { return (v + 255) / 256 * 256; }

struct PrefillLayout {
  int64_t P, sf_rows;
  size_t eo, bso, dst2src, src2dst, xq, xsf, hq, hsf, c2, gemm, total;
};

PrefillLayout prefill_layout(int64_t M, int64_t topk, int64_t H, int64_t I, int64_t E) {
  PrefillLayout l;
  l.P = M * topk;
  l.sf_rows = (l.P + 127) / 128 * 128 + 128 * E;
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t here = at;
    at += part(bytes);
    return here;
  };
  l.eo = take((size_t)(E + 1) * 4);
  l.bso = take((size_t)(E + 1) * 4);
  l.dst2src = take((size_t)l.P * 4);
  l.src2dst = take((size_t)l.P * 4);
  l.xq = take((size_t)l.P * H / 2);
  l.xsf = take(stage_sf_bytes(l.sf_rows, H));
  l.hq = take((size_t)l.P * I / 2);
  l.hsf = take((size_t)l.sf_rows * ((I / 16 + 3) / 4 * 4));
  l.c2 = take((size_t)l.P * H * 2);
  l.gemm = take(b200fp4_grouped_gemm_workspace_bytes(l.P, E));
  l.total = at;
  return l;
}

int permute_check(const int32_t* topk_ids, const int32_t* expert_map, int64_t global_E, int64_t M, int64_t topk, int64_t E,
                  const int32_t* expert_offsets, const int32_t* blockscale_offsets, const int32_t* dst2src, const int32_t* src2dst) {
  if (M < 0 || topk <= 0 || E <= 0 || E > kGroupMaxExperts || M * topk > (1 << 24)) return B200FP4_STATUS_INVALID_VALUE;
  if (!expert_offsets || !blockscale_offsets) return B200FP4_STATUS_INVALID_VALUE;
  if (M > 0 && (!topk_ids || !dst2src || !src2dst)) return B200FP4_STATUS_INVALID_VALUE;
  if (expert_map && global_E <= 0) return B200FP4_STATUS_INVALID_VALUE;
  return B200FP4_STATUS_SUCCESS;
}

int unpermute_check(const void* expert_out, int dtype, const int32_t* src2dst, const float* topk_weights, int64_t M, int64_t topk,
                    int64_t H, const void* out) {
  if (M < 0 || topk <= 0 || H <= 0 || (H % 2) != 0 || M > 65535) return B200FP4_STATUS_INVALID_VALUE;
  if (dtype != B200FP4_DTYPE_BF16 && dtype != B200FP4_DTYPE_F16) return B200FP4_STATUS_NOT_SUPPORTED;
  if (M > 0 && (!expert_out || !src2dst || !topk_weights || !out)) return B200FP4_STATUS_INVALID_VALUE;
  return B200FP4_STATUS_SUCCESS;
}

}  // namespace

void launch_moe_route(const int32_t* topk_ids, int P, const int32_t* expert_map, int global_E, int E, int32_t* expert_offsets,
                      int32_t* blockscale_offsets, int32_t* dst2src, int32_t* src2dst, void* tile_ws, cudaStream_t st) {
  launch_pdl(moe_route_kernel, dim3(kRouteBlocks), dim3(kRouteThreads), 0, st, topk_ids, P, expert_map, global_E, E, expert_offsets,
             blockscale_offsets, dst2src, src2dst, tile_ws ? grouped_hdr(tile_ws) : nullptr, tile_ws ? grouped_tiles(tile_ws) : nullptr,
             tile_ws ? grouped_max_tiles(P, E) : 0);
}

}  // namespace b200fp4

using namespace b200fp4;

extern "C" int b200fp4_moe_permute(const int32_t* topk_ids, const int32_t* expert_map, int64_t global_E, int64_t M,
                                   int64_t topk, int64_t E, int32_t* expert_offsets, int32_t* blockscale_offsets,
                                   int32_t* dst2src, int32_t* src2dst, void* stream) {
  const int refused = permute_check(topk_ids, expert_map, global_E, M, topk, E, expert_offsets, blockscale_offsets, dst2src, src2dst);
  if (refused != B200FP4_STATUS_SUCCESS) return refused;
  const int P = (int)(M * topk);
  cudaStream_t st = (cudaStream_t)stream;
  if (P <= kRouteMaxPairs) {
    launch_moe_route(topk_ids, P, expert_map, (int)global_E, (int)E, expert_offsets, blockscale_offsets, dst2src, src2dst, nullptr, st);
    return finish_launch(1);
  }
  if (cudaMemsetAsync(expert_offsets, 0, (size_t)(E + 1) * sizeof(int32_t), st) != cudaSuccess)
    return B200FP4_STATUS_EXECUTION_FAILED;
  const int blocks = (P + kPermuteBlock - 1) / kPermuteBlock;
  moe_permute_count_kernel<<<blocks, kPermuteBlock, 0, st>>>(topk_ids, P, expert_map, (int)global_E, (int)E,
                                                             expert_offsets, dst2src, src2dst);
  moe_permute_scan_kernel<<<1, 1024, 0, st>>>((int)E, expert_offsets, blockscale_offsets);
  moe_permute_scatter_kernel<<<blocks, kPermuteBlock, 0, st>>>(P, (int)E, expert_offsets, dst2src, src2dst);
  moe_permute_shift_kernel<<<1, 1024, 0, st>>>((int)E, expert_offsets);
  return finish_launch(4);
}

extern "C" int b200fp4_moe_unpermute_reduce(const void* expert_out, int dtype, const int32_t* src2dst,
                                            const float* topk_weights, int64_t M, int64_t topk, int64_t H, void* out,
                                            void* stream) {
  const int refused = unpermute_check(expert_out, dtype, src2dst, topk_weights, M, topk, H, out);
  if (refused != B200FP4_STATUS_SUCCESS || M == 0) return refused;
  if ((H % 8) == 0 && aligned(expert_out, 16) && aligned(out, 16)) {
    const dim3 grid8((unsigned)((H / 8 + kUnpermuteThreads - 1) / kUnpermuteThreads), (unsigned)M);
    if (dtype == B200FP4_DTYPE_BF16)
      launch_pdl(unpermute_reduce_vec8_kernel<__nv_bfloat16>, grid8, dim3(kUnpermuteThreads), 0, (cudaStream_t)stream,
                 reinterpret_cast<const __nv_bfloat16*>(expert_out), src2dst, topk_weights, (int)M, (int)topk, (int)H,
                 reinterpret_cast<__nv_bfloat16*>(out));
    else
      launch_pdl(unpermute_reduce_vec8_kernel<__half>, grid8, dim3(kUnpermuteThreads), 0, (cudaStream_t)stream,
                 reinterpret_cast<const __half*>(expert_out), src2dst, topk_weights, (int)M, (int)topk, (int)H,
                 reinterpret_cast<__half*>(out));
    return finish_launch(1);
  }
  dim3 grid((unsigned)((H / 2 + 127) / 128), (unsigned)M);
  if (dtype == B200FP4_DTYPE_BF16)
    unpermute_reduce_kernel<__nv_bfloat16><<<grid, 128, 0, (cudaStream_t)stream>>>(
        reinterpret_cast<const __nv_bfloat16*>(expert_out), src2dst, topk_weights, (int)M, (int)topk, (int)H,
        reinterpret_cast<__nv_bfloat16*>(out));
  else
    unpermute_reduce_kernel<__half><<<grid, 128, 0, (cudaStream_t)stream>>>(
        reinterpret_cast<const __half*>(expert_out), src2dst, topk_weights, (int)M, (int)topk, (int)H,
        reinterpret_cast<__half*>(out));
  return finish_launch(1);
}

extern "C" size_t b200fp4_moe_prefill_workspace_bytes(int64_t M, int64_t topk, int64_t H, int64_t I, int64_t E) {
  if (M <= 0 || topk <= 0 || H <= 0 || I <= 0 || E <= 0) return 0;
  return prefill_layout(M, topk, H, I, E).total;
}

extern "C" int b200fp4_moe_prefill(const void* hidden, int dtype, const float* topk_weights, const int32_t* topk_ids,
                                   const int32_t* expert_map, int64_t global_E, const void* w13_codes, const void* w13_sf,
                                   const float* alpha1, const void* w2_codes, const void* w2_sf, const float* alpha2,
                                   const float* a1_gs, const float* a2_gs, void* out, int64_t M, int64_t topk, int64_t H, int64_t I,
                                   int64_t E, void* workspace, size_t workspace_bytes, void* gemm_workspace, void* stream) {
  if (M < 0 || topk <= 0 || topk > 32 || H <= 0 || H % 64 != 0 || I <= 0 || I % 128 != 0 || E <= 0) return B200FP4_STATUS_INVALID_VALUE;
  if (M == 0) return B200FP4_STATUS_SUCCESS;
  const PrefillLayout l = prefill_layout(M, topk, H, I, E);
  if (!workspace || !aligned(workspace, 256) || workspace_bytes < l.total) return B200FP4_STATUS_ALLOC_FAILED;
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  int32_t* eo = reinterpret_cast<int32_t*>(ws + l.eo);
  int32_t* bso = reinterpret_cast<int32_t*>(ws + l.bso);
  int32_t* dst2src = reinterpret_cast<int32_t*>(ws + l.dst2src);
  int32_t* src2dst = reinterpret_cast<int32_t*>(ws + l.src2dst);
  const size_t gemm_bytes = b200fp4_grouped_gemm_workspace_bytes(l.P, E);
  unsigned char* gemm_ws = gemm_workspace ? static_cast<unsigned char*>(gemm_workspace) : ws + l.gemm;
  if (!aligned(gemm_ws, 16)) return B200FP4_STATUS_ALLOC_FAILED;
  // what any of the five steps would refuse, before the first of them is queued
  int rc = permute_check(topk_ids, expert_map, global_E, M, topk, E, eo, bso, dst2src, src2dst);
  if (rc == B200FP4_STATUS_SUCCESS)
    rc = experts_quantize_scatter_check(hidden, dtype, M, H, topk, src2dst, a1_gs, eo, bso, (int32_t)E, l.sf_rows, topk_ids, expert_map,
                                        global_E, ws + l.xq, ws + l.xsf, true);
  if (rc == B200FP4_STATUS_SUCCESS)
    rc = grouped_gemm_check(ws + l.xq, w13_codes, ws + l.xsf, w13_sf, alpha1, eo, bso, ws + l.hq, dtype, l.P, 2 * I, H, E, 0, gemm_ws,
                            gemm_bytes, ws + l.hsf, a2_gs, true);
  if (rc == B200FP4_STATUS_SUCCESS)
    rc = grouped_gemm_check(ws + l.hq, w2_codes, ws + l.hsf, w2_sf, alpha2, eo, bso, ws + l.c2, dtype, l.P, H, I, E, 0, gemm_ws, gemm_bytes,
                            nullptr, nullptr, false);
  if (rc == B200FP4_STATUS_SUCCESS) rc = unpermute_check(ws + l.c2, dtype, src2dst, topk_weights, M, topk, H, out);
  if (rc != B200FP4_STATUS_SUCCESS) return rc;
  if (b200fp4_has_hardware_acceleration() != 1) return B200FP4_STATUS_ARCH_MISMATCH;
  cudaStream_t st = (cudaStream_t)stream;
  const bool one_launch = l.P <= kRouteMaxPairs;                   // metadata and tile list together
  if (one_launch) {
    launch_moe_route(topk_ids, (int)l.P, expert_map, (int)global_E, (int)E, eo, bso, nullptr, src2dst, gemm_ws, st);
    rc = finish_launch(1);
  } else {
    rc = b200fp4_moe_permute(topk_ids, expert_map, global_E, M, topk, E, eo, bso, dst2src, src2dst, stream);
  }
  if (rc == B200FP4_STATUS_SUCCESS)
    rc = experts_quantize_scatter(hidden, dtype, M, H, topk, src2dst, a1_gs, eo, bso, (int32_t)E, l.sf_rows, topk_ids, expert_map, global_E,
                                  ws + l.xq, ws + l.xsf, stream, true);
  if (rc == B200FP4_STATUS_SUCCESS)
    rc = grouped_gemm(ws + l.xq, w13_codes, ws + l.xsf, w13_sf, alpha1, eo, bso, ws + l.hq, dtype, l.P, 2 * I, H, E, 0, gemm_ws,
                      gemm_bytes, stream, ws + l.hsf, a2_gs, one_launch, true);
  if (rc == B200FP4_STATUS_SUCCESS)
    rc = grouped_gemm(ws + l.hq, w2_codes, ws + l.hsf, w2_sf, alpha2, eo, bso, ws + l.c2, dtype, l.P, H, I, E, 0, gemm_ws, gemm_bytes,
                      stream, nullptr, nullptr, true, false);
  if (rc == B200FP4_STATUS_SUCCESS)
    rc = b200fp4_moe_unpermute_reduce(ws + l.c2, dtype, src2dst, topk_weights, M, topk, H, out, stream);
  return rc;
}
