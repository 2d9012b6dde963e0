// bf16/f16 -> NVFP4 quantizer for sm_100a.
//
// Plain tensors (quantize_rows_kernel): one thread owns the 16 elements of a scale block, four of them in rows 32 apart.
// Permuted rows with a scale per expert (quantize_kernel): one thread owns 8 consecutive elements (one 16-byte load); two
// neighbouring lanes form a scale block and share the block maximum (found with packed 16-bit max) through a warp shuffle.
// Arithmetic follows ref_nvfp4_quant (vllm/model_executor/layers/quantization/utils/
// nvfp4_emulation_utils.py:439-453) operation by operation in IEEE fp32 -- explicit _rn
// intrinsics keep the compiler from contracting or approximating -- so codes and scales are
// bit-identical to the reference's emulation path; the E2M1 rounding itself is the native
// cvt.rn.satfinite.e2m1x2.f32 that replaces the reference's software routine
// (patch_nvfp4_utils_sw_e2m1.py:31-63).
#include "grouped.cuh"
#include "quant.cuh"

namespace b200fp4 {

std::atomic<uint64_t> g_launch_count{0};

namespace {

constexpr int kTX = 64;    // threads along K (each 8 elements): 512 elements per block row
constexpr int kTY = 4;     // rows per block per pass
constexpr int kRows = 4;   // passes (rows) per thread, loads issued together

// One global scale for the tensor.  Bound by HBM (2.5625 bytes per element); what it takes to get near that:
//   * a thread owns whole blocks of 16 (32-byte loads, no shuffle for the maximum, the scale arithmetic once per block and no
//     table to fill first) and has four in flight, in rows m, m+32, m+64, m+96 of a 128-row tile;
//   * the scale bytes of those four rows and four neighbouring lanes are 16 contiguous bytes of the swizzled layout, one store
//     (a store per byte before), and rows m and m+1 of a block complete the sector;
//   * rows past M and blocks past K write zero scales here, so that no memset goes ahead of the kernel.
// Measured: see the launch code.
constexpr int kQrThreads = 256;
constexpr int kQrRows = 4;                   // rows of a thread, 32 apart
enum { kQrLoad32 = 1, kQrStore8 = 2, kQrSfWide = 4 };      // alignment the pointers and strides allow

template <typename T, bool kSwizzled>
__global__ void __launch_bounds__(kQrThreads, 4)
    quantize_rows_kernel(const T* __restrict__ x, int64_t M, int KB, int64_t ldx, const float* __restrict__ gs_ptr,
                         uint8_t* __restrict__ codes, uint8_t* __restrict__ sf, int align) {
  pdl_wait();
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kb = blockIdx.x * 32 + lane;       // block of 16 along K
  const int KT = (KB + 3) >> 2;
  const int64_t m0 = (int64_t)(blockIdx.y >> 2) * 128 + (blockIdx.y & 3) * 8 + warp;
  const bool col_ok = kb < KB;
  uint4 r0[kQrRows], r1[kQrRows];
#pragma unroll
  for (int i = 0; i < kQrRows; ++i) {
    r0[i] = r1[i] = make_uint4(0, 0, 0, 0);
    const int64_t m = m0 + 32 * i;
    if (col_ok && m < M) {
      const T* p = x + m * ldx + (int64_t)kb * 16;
      if (align & kQrLoad32) {
        ldg_stream_v8(p, r0[i], r1[i]);
      } else {
        r0[i] = ldg_stream_u4(p);
        r1[i] = ldg_stream_u4(p + 8);
      }
    }
  }
  const float gs = gs_ptr[0];
  const float rcp_gs = __frcp_rn(gs + (gs == 0.f ? 1.0e8f : 0.f));
  uint32_t sfw[kQrRows];
#pragma unroll
  for (int i = 0; i < kQrRows; ++i) {
    const int64_t m = m0 + 32 * i;
    const bool ok = col_ok && m < M;
    uint32_t sfb;
    const uint2 c = quantize_block16<T>(r0[i], r1[i], gs, [&](uint32_t b) { return out_scale_of((uint8_t)b, rcp_gs); }, sfb);
    if (!ok) sfb = 0;
    if (ok) {
      uint8_t* dst = codes + (m * KB + kb) * 8;
      if (align & kQrStore8) {
        *reinterpret_cast<uint2*>(dst) = c;
      } else {
        reinterpret_cast<uint32_t*>(dst)[0] = c.x;
        reinterpret_cast<uint32_t*>(dst)[1] = c.y;
      }
    }
    if (align & kQrSfWide) {
      sfw[i] = sfb << (8 * (lane & 3));        // four lanes put their bytes together
      sfw[i] |= __shfl_xor_sync(0xffffffffu, sfw[i], 1);
      sfw[i] |= __shfl_xor_sync(0xffffffffu, sfw[i], 2);
      if (!kSwizzled && (lane & 3) == 0 && ok) *reinterpret_cast<uint32_t*>(sf + m * KB + kb) = sfw[i];
    } else if (kSwizzled) {
      if (kb < 4 * KT) sf[sf_swizzled_offset(m, kb, KT)] = (uint8_t)sfb;
    } else if (ok) {
      sf[m * KB + kb] = (uint8_t)sfb;
    }
  }
  if (kSwizzled && (align & kQrSfWide) && (lane & 3) == 0 && kb < 4 * KT)
    *reinterpret_cast<uint4*>(sf + sf_swizzled_offset(m0, kb, KT)) = make_uint4(sfw[0], sfw[1], sfw[2], sfw[3]);
}

// Rows grouped by expert: per-row expert lookup (global scale + scale-factor row offset per expert), swizzled scales.
// kSilu: input is [M, 2K]; quantize round_to_T(silu(x[:, :K]) * x[:, K:]).
template <typename T, bool kSilu>
__global__ void __launch_bounds__(kTX* kTY)
    quantize_kernel(const T* __restrict__ x, int64_t M, int64_t K, int64_t ldx, const float* __restrict__ gs_ptr,
                    const int32_t* __restrict__ expert_offsets, const int32_t* __restrict__ blockscale_offsets,
                    int num_experts, uint8_t* __restrict__ codes, uint8_t* __restrict__ sf,
                    const int32_t* __restrict__ row_map, int row_div) {
  const int64_t kc = (int64_t)blockIdx.x * kTX + threadIdx.x;  // 8-element chunk index along K
  const int64_t CPR = K >> 3;
  const int64_t KT = ((K >> 4) + 3) >> 2;
  const int64_t m0 = ((int64_t)blockIdx.y * kTY + threadIdx.y) * kRows;
  const bool col_ok = kc < CPR;

  uint4 raw[kRows], raw2[kRows];
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    raw[r] = make_uint4(0, 0, 0, 0);
    raw2[r] = make_uint4(0, 0, 0, 0);
    const int64_t m = m0 + r;
    if (col_ok && m < M) {
      // optional gather: output row m is source row row_map[m] / row_div (a negative entry reads as zeros)
      int64_t src = m;
      if (row_map != nullptr) {
        const int v = row_map[m];
        src = v < 0 ? -1 : (int64_t)(v / row_div);
      }
      if (src >= 0) {
        raw[r] = *reinterpret_cast<const uint4*>(x + src * ldx + kc * 8);
        if (kSilu) raw2[r] = *reinterpret_cast<const uint4*>(x + src * ldx + K + kc * 8);
      }
    }
  }

  // The block's 16 rows look their expert up once each (not once per thread):
  // global scale, its guarded reciprocal and the row of the scale-factor tensor.
  __shared__ float s_gs[kTY * kRows], s_rcp[kTY * kRows];
  __shared__ long long s_sfrow[kTY * kRows];
  {
    const int t = threadIdx.y * kTX + threadIdx.x;
    if (t < kTY * kRows) {
      // slot t = (threadIdx.y = t / kRows, pass r = t % kRows) holds row (blockIdx.y * kTY + t / kRows) * kRows + t % kRows
      const int64_t m = ((int64_t)blockIdx.y * kTY + t / kRows) * kRows + t % kRows;
      float gs = 0.f;
      long long row = m;
      if (m < M) {
        int lo = 0, hi = num_experts - 1;      // largest e with expert_offsets[e] <= m
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if ((int64_t)expert_offsets[mid] <= m) lo = mid;
          else hi = mid - 1;
        }
        gs = gs_ptr[lo];
        row = (long long)blockscale_offsets[lo] + (m - (long long)expert_offsets[lo]);
      }
      s_gs[t] = gs;
      s_rcp[t] = __frcp_rn(gs + (gs == 0.f ? 1.0e8f : 0.f));
      s_sfrow[t] = row;
    }
    __syncthreads();
  }

#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    const int64_t m = m0 + r;
    const bool ok = col_ok && m < M;
    float v[8];
    float amax;
    if (kSilu) {
      float u[8];
      unpack8<T>(raw[r], v);
      unpack8<T>(raw2[r], u);
      amax = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        v[i] = to_f32<T>(from_f32<T>(silu_f32(v[i]) * u[i]));
        amax = fmaxf(amax, fabsf(v[i]));
      }
    } else {
      amax = amax8<T>(raw[r]);
      unpack8<T>(raw[r], v);
    }
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));

    const float gs = s_gs[threadIdx.y * kRows + r];
    const int64_t sf_row = s_sfrow[threadIdx.y * kRows + r];

    float scale = __fmul_rn(gs, __fmul_rn(amax, 0.16666667163372039794921875f));  // fl32(1/6)
    scale = fminf(scale, 448.f);
    const uint8_t sfb = f32_to_e4m3(scale);
    const float os = out_scale_of(sfb, s_rcp[threadIdx.y * kRows + r]);

    const uint32_t packed =
        f32x8_to_e2m1(__fmul_rn(v[0], os), __fmul_rn(v[1], os), __fmul_rn(v[2], os), __fmul_rn(v[3], os),
                      __fmul_rn(v[4], os), __fmul_rn(v[5], os), __fmul_rn(v[6], os), __fmul_rn(v[7], os));
    if (ok) {
      *reinterpret_cast<uint32_t*>(codes + m * (K >> 1) + kc * 4) = packed;
      if ((kc & 1) == 0) sf[sf_swizzled_offset(sf_row, kc >> 1, KT)] = sfb;
    }
  }
}

// Token-major form of the gather above: block t reads source row t once and quantizes it for each of its
// `topk` destination rows src2dst[t*topk + s] (negative = no destination), each with the global scale of the
// expert that owns the destination row.  Same bytes as quantizing the gathered rows one by one; the source is
// read once instead of topk times.
// One thread = one block of 16 elements (the block maximum needs no other lane, the scale arithmetic is done once): with two
// lanes per block the kernel issued 70 instructions per 8 elements and destination and was bound by that (8192 x 2048, ten
// destinations: 51-58 us, 82 % of the issue slots).  Slots whose expert has the global scale of the slot before share its
// codes -- the arithmetic depends on nothing else -- and only store them again.  Four lanes put their scale bytes together for
// one 4-byte store; with kStageSf (the grouped GEMM's own layout) sixteen lanes for one of 16 bytes: the 4-byte stores, each to
// a sector of its own, were half of all sectors written (8192 x 2048, ten destinations: 45.3 us, 35.5 so, 33.2 without scales).
constexpr int kScatterMaxTopk = 32;
constexpr int kScatterThreads = 256;

template <typename T, bool kStageSf>
__global__ void __launch_bounds__(kScatterThreads)
    experts_quantize_scatter_kernel(const T* __restrict__ x, int64_t K, int topk, const int32_t* __restrict__ src2dst,
                                    const float* __restrict__ gs_ptr, const int32_t* __restrict__ expert_offsets,
                                    const int32_t* __restrict__ blockscale_offsets, int num_experts,
                                    const int32_t* __restrict__ topk_ids, const int32_t* __restrict__ expert_map,
                                    int global_E, uint8_t* __restrict__ codes, uint8_t* __restrict__ sf) {
  __shared__ float s_gs[kScatterMaxTopk], s_rcp[kScatterMaxTopk];
  __shared__ long long s_sfrow[kScatterMaxTopk], s_code[kScatterMaxTopk];
  __shared__ int s_dst[kScatterMaxTopk];
  pdl_wait();
  pdl_launch_dependents();
  const int64_t t = blockIdx.x;
  const int KB = (int)(K >> 4);
  const int64_t KT = (KB + 3) >> 2;
  const T* row_src = x + t * K;
  // the first piece of the row is requested before the destination lookup, so the two latencies overlap
  uint4 r0 = make_uint4(0, 0, 0, 0), r1 = r0;
  if ((int)threadIdx.x < KB) {
    r0 = reinterpret_cast<const uint4*>(row_src)[2 * threadIdx.x];
    r1 = reinterpret_cast<const uint4*>(row_src)[2 * threadIdx.x + 1];
  }
  if ((int)threadIdx.x < topk) {
    const int dst = src2dst[t * topk + threadIdx.x];
    float gs = 0.f;
    long long row = 0;
    if (dst >= 0) {
      int lo;
      if (topk_ids != nullptr) {
        // the pair's routing entry names the expert directly
        lo = topk_ids[t * topk + threadIdx.x];
        if (expert_map != nullptr) lo = (lo >= 0 && lo < global_E) ? expert_map[lo] : 0;
        lo = min(max(lo, 0), num_experts - 1);
      } else {
        lo = 0;
        int hi = num_experts - 1;            // largest e with expert_offsets[e] <= dst
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (expert_offsets[mid] <= dst) lo = mid;
          else hi = mid - 1;
        }
      }
      gs = gs_ptr[lo];
      row = (long long)blockscale_offsets[lo] + (dst - expert_offsets[lo]);
    }
    s_dst[threadIdx.x] = dst;
    s_gs[threadIdx.x] = gs;
    s_rcp[threadIdx.x] = __frcp_rn(gs + (gs == 0.f ? 1.0e8f : 0.f));
    // byte offsets of the destination row in the code tensor and of its first scale byte, computed once per block
    s_sfrow[threadIdx.x] = kStageSf ? (row >> 7) * ((KB + 15) >> 4) * 2048 + (row & 127) * 16 : sf_swizzled_offset(row, 0, KT);
    s_code[threadIdx.x] = (long long)dst * (long long)(K >> 1);
  }
  __syncthreads();
  const bool sf_words = (KB & 3) == 0;         // the four lanes of a scale word are then all inside the row
  for (int kb0 = 0; kb0 < KB; kb0 += blockDim.x) {
    const int kb = kb0 + threadIdx.x;
    const bool ok = kb < KB;
    if (kb0 > 0 && ok) {
      r0 = reinterpret_cast<const uint4*>(row_src)[2 * kb];
      r1 = reinterpret_cast<const uint4*>(row_src)[2 * kb + 1];
    }
    float v[16];
    unpack8<T>(r0, v);
    unpack8<T>(r1, v + 8);
    const float sixth = __fmul_rn(fmaxf(amax8<T>(r0), amax8<T>(r1)), 0.16666667163372039794921875f);
    // scale byte of this block of 16 relative to its row's first
    const int64_t sf_col = kStageSf ? (int64_t)(kb >> 4) * 2048 + (kb & 15) : (int64_t)(kb >> 2) * 512 + (kb & 3);
    uint2 packed = make_uint2(0, 0);
    uint32_t sfb = 0, sf4 = 0;
    uint4 sf16 = make_uint4(0, 0, 0, 0);
    float last_gs = __int_as_float(0x7FFFFFFF);                     // a NaN: equal to nothing
    for (int sl = 0; sl < topk; ++sl) {
      if (s_dst[sl] < 0) continue;
      const float gs = s_gs[sl];
      if (gs != last_gs) {
        last_gs = gs;
        sfb = f32_to_e4m3(fminf(__fmul_rn(gs, sixth), 448.f));
        const float os = out_scale_of((uint8_t)sfb, s_rcp[sl]);
        packed.x = f32x8_to_e2m1(__fmul_rn(v[0], os), __fmul_rn(v[1], os), __fmul_rn(v[2], os), __fmul_rn(v[3], os),
                                 __fmul_rn(v[4], os), __fmul_rn(v[5], os), __fmul_rn(v[6], os), __fmul_rn(v[7], os));
        packed.y = f32x8_to_e2m1(__fmul_rn(v[8], os), __fmul_rn(v[9], os), __fmul_rn(v[10], os), __fmul_rn(v[11], os),
                                 __fmul_rn(v[12], os), __fmul_rn(v[13], os), __fmul_rn(v[14], os), __fmul_rn(v[15], os));
        sf4 = sfb << (8 * (threadIdx.x & 3));
        sf4 |= __shfl_xor_sync(0xffffffffu, sf4, 1);
        sf4 |= __shfl_xor_sync(0xffffffffu, sf4, 2);
        if (kStageSf)
          sf16 = make_uint4(sf4, __shfl_down_sync(0xffffffffu, sf4, 4), __shfl_down_sync(0xffffffffu, sf4, 8),
                            __shfl_down_sync(0xffffffffu, sf4, 12));
      }
      if (ok) {
        *reinterpret_cast<uint2*>(codes + s_code[sl] + kb * 8) = packed;
        if (kStageSf) {
          if ((threadIdx.x & 15) == 0) *reinterpret_cast<uint4*>(sf + s_sfrow[sl] + sf_col) = sf16;
        } else if (!sf_words) sf[s_sfrow[sl] + sf_col] = (uint8_t)sfb;
        else if ((threadIdx.x & 3) == 0) *reinterpret_cast<uint32_t*>(sf + s_sfrow[sl] + sf_col) = sf4;
      }
    }
  }
}

template <typename T, bool kSilu>
void launch(const void* x, int64_t M, int64_t K, int64_t ldx, const float* gs, const int32_t* eo, const int32_t* bo,
            int ne, void* codes, void* sf, cudaStream_t st, const int32_t* row_map, int row_div) {
  dim3 block(kTX, kTY);
  dim3 grid((unsigned)(((K >> 3) + kTX - 1) / kTX), (unsigned)((M + kTY * kRows - 1) / (kTY * kRows)));
  quantize_kernel<T, kSilu><<<grid, block, 0, st>>>(reinterpret_cast<const T*>(x), M, K, ldx, gs, eo, bo, ne, (uint8_t*)codes,
                                                    (uint8_t*)sf, row_map, row_div);
}

// 16384 x 4096 bf16: 37.1 us with 8 elements per thread and a table per block (4.6 TB/s), 29 us so (5.9 TB/s of 6.55).
template <typename T>
void launch_rows(const void* x, int64_t M, int64_t KB, int64_t ldx, const float* gs, void* codes, void* sf, bool swizzled, cudaStream_t st) {
  int align = (aligned(x, 32) && ldx % 16 == 0 ? kQrLoad32 : 0) | (aligned(codes, 8) ? kQrStore8 : 0);
  if (swizzled ? aligned(sf, 16) : (aligned(sf, 4) && KB % 4 == 0)) align |= kQrSfWide;
  // whole 128-row tiles where the padding rows' scales have to be written
  const int64_t row_blocks = swizzled ? (M + 127) / 128 * 4 : (M / 128) * 4 + (M % 128 < 32 ? (M % 128 + 7) / 8 : 4);
  const dim3 grid((unsigned)((KB + 31) / 32), (unsigned)row_blocks);
  if (swizzled)
    launch_pdl(quantize_rows_kernel<T, true>, grid, dim3(kQrThreads), 0, st, static_cast<const T*>(x), M, (int)KB, ldx, gs,
               (uint8_t*)codes, (uint8_t*)sf, align);
  else
    launch_pdl(quantize_rows_kernel<T, false>, grid, dim3(kQrThreads), 0, st, static_cast<const T*>(x), M, (int)KB, ldx, gs,
               (uint8_t*)codes, (uint8_t*)sf, align);
}

}  // namespace
}  // namespace b200fp4

using namespace b200fp4;

extern "C" size_t b200fp4_sf_swizzled_bytes(int64_t rows, int64_t k_blocks) {
  if (rows < 0 || k_blocks < 0) return 0;
  return (size_t)(((rows + 127) / 128) * 128 * (((k_blocks + 3) / 4) * 4));
}

int b200fp4::quantize_check(const void* x, int in_dtype, int64_t M, int64_t K, int64_t ldx, const float* global_scale, const void* codes,
                            const void* sf) {
  if (M < 0 || K <= 0 || (K % 16) != 0 || ldx < K || (ldx % 8) != 0) return B200FP4_STATUS_INVALID_VALUE;
  if (in_dtype != B200FP4_DTYPE_F16 && in_dtype != B200FP4_DTYPE_BF16) return B200FP4_STATUS_NOT_SUPPORTED;
  if (M == 0) return B200FP4_STATUS_SUCCESS;
  if (!x || !global_scale || !codes || !sf) return B200FP4_STATUS_INVALID_VALUE;
  if (!aligned(x, 16) || !aligned(codes, 4)) return B200FP4_STATUS_INVALID_VALUE;
  if (M > (int64_t)65535 * kTY * kRows || K > ((int64_t)1 << 30)) return B200FP4_STATUS_NOT_SUPPORTED;
  return B200FP4_STATUS_SUCCESS;
}

extern "C" int b200fp4_quantize(const void* x, int in_dtype, int64_t M, int64_t K, int64_t ldx,
                                const float* global_scale, void* codes, void* sf, int sf_swizzled, void* stream) {
  const int refused = quantize_check(x, in_dtype, M, K, ldx, global_scale, codes, sf);
  if (refused != B200FP4_STATUS_SUCCESS || M == 0) return refused;
  cudaStream_t st = (cudaStream_t)stream;
  if (in_dtype == B200FP4_DTYPE_BF16)
    launch_rows<__nv_bfloat16>(x, M, K / 16, ldx, global_scale, codes, sf, sf_swizzled != 0, st);
  else
    launch_rows<__half>(x, M, K / 16, ldx, global_scale, codes, sf, sf_swizzled != 0, st);
  return finish_launch(1);
}

static int experts_quantize_impl(const void* x, int in_dtype, int64_t M, int64_t K, const float* global_scales,
                                 const int32_t* expert_offsets, const int32_t* blockscale_offsets, int32_t num_experts,
                                 int64_t sf_rows_padded, int silu_mul, void* codes, void* sf, void* stream,
                                 const int32_t* row_map, int row_div) {
  if (M < 0 || K <= 0 || (K % 16) != 0 || num_experts <= 0 || sf_rows_padded < 0 || (sf_rows_padded % 128) != 0)
    return B200FP4_STATUS_INVALID_VALUE;
  if (in_dtype != B200FP4_DTYPE_F16 && in_dtype != B200FP4_DTYPE_BF16) return B200FP4_STATUS_NOT_SUPPORTED;
  if (!global_scales || !expert_offsets || !blockscale_offsets || !sf) return B200FP4_STATUS_INVALID_VALUE;
  if (M > 0 && (!x || !codes || !aligned(x, 16) || !aligned(codes, 4))) return B200FP4_STATUS_INVALID_VALUE;
  if (M > (int64_t)65535 * kTY * kRows) return B200FP4_STATUS_NOT_SUPPORTED;
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t KB = K / 16;
  if (cudaMemsetAsync(sf, 0, (size_t)(sf_rows_padded * (((KB + 3) / 4) * 4)), st) != cudaSuccess) {
    cudaGetLastError();
    return B200FP4_STATUS_EXECUTION_FAILED;
  }
  if (M == 0) return finish_launch(1);
  const bool bf = in_dtype == B200FP4_DTYPE_BF16;
  const int64_t ldx = silu_mul ? 2 * K : K;
  if (silu_mul) {
    if (bf) launch<__nv_bfloat16, true>(x, M, K, ldx, global_scales, expert_offsets, blockscale_offsets, num_experts, codes, sf, st, row_map, row_div);
    else launch<__half, true>(x, M, K, ldx, global_scales, expert_offsets, blockscale_offsets, num_experts, codes, sf, st, row_map, row_div);
  } else {
    if (bf) launch<__nv_bfloat16, false>(x, M, K, ldx, global_scales, expert_offsets, blockscale_offsets, num_experts, codes, sf, st, row_map, row_div);
    else launch<__half, false>(x, M, K, ldx, global_scales, expert_offsets, blockscale_offsets, num_experts, codes, sf, st, row_map, row_div);
  }
  return finish_launch(2);
}

extern "C" int b200fp4_experts_quantize(const void* x, int in_dtype, int64_t M, int64_t K, const float* global_scales,
                                        const int32_t* expert_offsets, const int32_t* blockscale_offsets,
                                        int32_t num_experts, int64_t sf_rows_padded, int silu_mul, void* codes,
                                        void* sf, void* stream) {
  return experts_quantize_impl(x, in_dtype, M, K, global_scales, expert_offsets, blockscale_offsets, num_experts,
                               sf_rows_padded, silu_mul, codes, sf, stream, nullptr, 1);
}

namespace b200fp4 {

int experts_quantize_scatter_check(const void* x, int in_dtype, int64_t n_src, int64_t K, int64_t topk, const int32_t* src2dst,
                                   const float* global_scales, const int32_t* expert_offsets, const int32_t* blockscale_offsets,
                                   int32_t num_experts, int64_t sf_rows_padded, const int32_t* topk_ids, const int32_t* expert_map,
                                   int64_t global_E, const void* codes, const void* sf, bool stage_sf) {
  if (expert_map && (!topk_ids || global_E <= 0)) return B200FP4_STATUS_INVALID_VALUE;
  if (n_src < 0 || K <= 0 || (K % 16) != 0 || topk <= 0 || num_experts <= 0 || sf_rows_padded < 0 ||
      (sf_rows_padded % 128) != 0)
    return B200FP4_STATUS_INVALID_VALUE;
  if (in_dtype != B200FP4_DTYPE_F16 && in_dtype != B200FP4_DTYPE_BF16) return B200FP4_STATUS_NOT_SUPPORTED;
  if (topk > kScatterMaxTopk || n_src > 0x7FFFFFFF) return B200FP4_STATUS_NOT_SUPPORTED;
  if (!global_scales || !expert_offsets || !blockscale_offsets || !sf) return B200FP4_STATUS_INVALID_VALUE;
  if (n_src > 0 && (!x || !codes || !src2dst || !aligned(x, 16) || !aligned(codes, 8) || !aligned(sf, 4)))
    return B200FP4_STATUS_INVALID_VALUE;
  if (stage_sf && ((K % 64) != 0 || !aligned(sf, 16))) return B200FP4_STATUS_INVALID_VALUE;
  return B200FP4_STATUS_SUCCESS;
}

int experts_quantize_scatter(const void* x, int in_dtype, int64_t n_src, int64_t K, int64_t topk, const int32_t* src2dst,
                             const float* global_scales, const int32_t* expert_offsets, const int32_t* blockscale_offsets,
                             int32_t num_experts, int64_t sf_rows_padded, const int32_t* topk_ids, const int32_t* expert_map,
                             int64_t global_E, void* codes, void* sf, void* stream, bool stage_sf) {
  const int refused = experts_quantize_scatter_check(x, in_dtype, n_src, K, topk, src2dst, global_scales, expert_offsets,
                                                     blockscale_offsets, num_experts, sf_rows_padded, topk_ids, expert_map, global_E,
                                                     codes, sf, stage_sf);
  if (refused != B200FP4_STATUS_SUCCESS) return refused;
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t KB = K / 16;
  if (!stage_sf && cudaMemsetAsync(sf, 0, (size_t)(sf_rows_padded * (((KB + 3) / 4) * 4)), st) != cudaSuccess) {
    cudaGetLastError();
    return B200FP4_STATUS_EXECUTION_FAILED;
  }
  if (n_src == 0) return finish_launch(1);
  const unsigned threads = (unsigned)(KB >= kScatterThreads ? kScatterThreads : (KB + 31) / 32 * 32);
  auto launch = [&](auto* kernel, const auto* src) {
    launch_pdl(kernel, dim3((unsigned)n_src), dim3(threads), 0, st, src, K, (int)topk, src2dst, global_scales, expert_offsets,
               blockscale_offsets, num_experts, topk_ids, expert_map, (int)global_E, (uint8_t*)codes, (uint8_t*)sf);
  };
  if (in_dtype == B200FP4_DTYPE_BF16)
    launch(stage_sf ? experts_quantize_scatter_kernel<__nv_bfloat16, true> : experts_quantize_scatter_kernel<__nv_bfloat16, false>,
           reinterpret_cast<const __nv_bfloat16*>(x));
  else
    launch(stage_sf ? experts_quantize_scatter_kernel<__half, true> : experts_quantize_scatter_kernel<__half, false>,
           reinterpret_cast<const __half*>(x));
  return finish_launch(stage_sf ? 1 : 2);
}

}  // namespace b200fp4

extern "C" int b200fp4_experts_quantize_scatter(const void* x, int in_dtype, int64_t n_src, int64_t K, int64_t topk,
                                                const int32_t* src2dst, const float* global_scales,
                                                const int32_t* expert_offsets, const int32_t* blockscale_offsets,
                                                int32_t num_experts, int64_t sf_rows_padded, const int32_t* topk_ids,
                                                const int32_t* expert_map, int64_t global_E, void* codes, void* sf,
                                                void* stream) {
  return experts_quantize_scatter(x, in_dtype, n_src, K, topk, src2dst, global_scales, expert_offsets, blockscale_offsets, num_experts,
                                  sf_rows_padded, topk_ids, expert_map, global_E, codes, sf, stream, false);
}

extern "C" int b200fp4_experts_quantize_gather(const void* x, int in_dtype, int64_t M, int64_t K, const float* global_scales,
                                               const int32_t* expert_offsets, const int32_t* blockscale_offsets,
                                               int32_t num_experts, int64_t sf_rows_padded, const int32_t* row_map,
                                               int32_t row_div, void* codes, void* sf, void* stream) {
  if (!row_map || row_div <= 0) return B200FP4_STATUS_INVALID_VALUE;
  return experts_quantize_impl(x, in_dtype, M, K, global_scales, expert_offsets, blockscale_offsets, num_experts,
                               sf_rows_padded, 0, codes, sf, stream, row_map, row_div);
}
