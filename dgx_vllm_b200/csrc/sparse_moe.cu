// 2:4-sparse NVFP4 batched GEMV and the fused MoE decode layer for sm_100a.
//
// Replaces sparse_fp4_kernel/sparse_fp4_v7.cu of the reference with a different execution plan:
//   * a "plan" kernel groups the (token, expert) pairs by expert and cuts them into passes of at
//     most four (or eight) tokens, so an expert's weights are streamed from HBM once per layer (per
//     pass) instead of once per pair;
//   * two persistent GEMV kernels (one block per SM) walk (pass, column slab) work items: the
//     tensor-core kernel further down (mma.sp; needs ordered metadata indices and one scale per 16 k)
//     and the general kernel described here, which takes any metadata.  In the general kernel a thread
//     owns 16 output columns and one K-slice.  Its weight bytes (four compressed rows, two
//     metadata rows, one scale row per 16 k) arrive through a private multi-stage cp.async ring in
//     shared memory that keeps running across work-item boundaries, so HBM latency is hidden
//     without holding prefetched data in registers;
//   * E2M1 byte -> half2 and metadata byte -> byte-permute selector decoding are table look-ups in
//     shared memory (32 copies per entry, one per bank: conflict free); the table index is built by
//     a single PRMT that merges the byte with the lane's bank offset;
//   * the 2:4 gather of the activation is one PRMT, products are packed half2 FMAs, and every
//     16-element scale block is folded into an fp32 accumulator;
//   * the K reduction is done in-kernel (warp shuffles, then one shared-memory pass), so there is
//     no partial-sum tensor and no separate reduction kernel; SiLU(gate)*up is fused into the
//     gate_up epilogue; the router-weighted sum is a small deterministic kernel (no atomics).
#include <cmath>
#include <type_traits>

#include <mutex>

#include "moe_small.cuh"
#include "sparse_mma.cuh"

extern "C" size_t b200fp4_sparse_workspace_bytes(int64_t P, int64_t K, int64_t E);

namespace b200fp4 {
namespace {

constexpr int kThreads = 256;      // block size of the 16-columns-per-thread variant
constexpr int kMaxTok = 4;       // tokens of one expert processed per pass over its weights
constexpr int kPlanThreads = 1024;
constexpr int kPlanMaxExperts = 4096;
constexpr int kLutBytes = 256 * 256;   // 256 rows of [32 x comp entry | 32 x meta entry]

struct Plan {
  int* hdr;        // [0] = number of unique experts, [1] = number of passes, [2] and [4] = work-item counters of the
                   // warp-scheduled GEMV (one per projection), [3] = status word of the one-launch layer
  int* pairs;      // [P]  pair indices grouped by expert
  int* mapped;     // [P]  local expert id of each pair, or -1
  int4* pass_rec;  // [passes][2]: {expert, n_tokens, pair0, pair1}, {pair2, pair3, index of pair0 in pairs[], -}
};

struct GemvArgs {
  SparseWeights w;
  Plan plan;
  const __half* A;  // [rows, K] fp16; the row of pair p is p / a_div
  int64_t lda;
  int a_div;
  uint32_t a_magic; // 0 if a_div == 1, else floor(2^32 / a_div) + 1: pair / a_div == umulhi(pair, a_magic) for pair < 2^16
  void* out;        // [P, N] (or [P, N/2] in SiLU mode), leading dimension ldo
  int64_t ldo;
  int out_dtype;
  int N, K;
  int n_slabs;
  int inter;        // SiLU mode: gate columns [0, inter), up columns [inter, 2*inter)
  long long wait_cycles;   // one-launch layer: clock64 budget of a wait on a pass counter
};

// ------------------------------------------------------------------------------------------ plan

// Activation copy modes of the plan kernel's extra blocks.
//   kConvBf16      bf16 -> fp16, same element order
//   kConvBf16Frag  bf16 -> fp16 in "fragment order" (below)
//   kConvF16Frag   fp16 copy in fragment order
// Fragment order: inside every group of 32 elements (16 words of two halves) word 4i + t is stored at position
// 4t + i (a 4 x 4 transpose of words).  The 16 bytes at offset 16t of a group are then exactly the four B-operand
// registers of lane t of a quad for one 32-wide k-step of mma.m16n8k32, which the warp-scheduled GEMV fetches with a
// single 16-byte asynchronous copy per lane.
enum { kConvNone = 0, kConvBf16 = 1, kConvBf16Frag = 2, kConvF16Frag = 3 };

__device__ __forceinline__ uint32_t bf16x2_to_f16x2(uint32_t w) {
  const __half2 h = __float22half2_rn(__bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w)));
  return *reinterpret_cast<const uint32_t*>(&h);
}


// The plan of few pairs, one pair per thread of the first eight warps: ranks by warp-wide matching, one warp after the other,
// and passes numbered by the first pair of their expert, so that nothing is as long as the number of experts (a decode step
// waits for this kernel from end to end: 4.6 us with the general path below, 2.7 us so at 10 pairs and 512 experts).
constexpr int kPlanSmallPairs = 256;
__device__ __forceinline__ void plan_small(const int32_t* __restrict__ ids, int P, const int32_t* __restrict__ expert_map, int global_E,
                                           int E, const Plan& plan, int ids_topk, int64_t ids_ld, int* zero_buf, int zero_count,
                                           int* s_count, int (*s_warp)[32]) {
  constexpr int kThr = kPlanSmallPairs;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid >= kThr) {                           // the other warps clear the counters and are done
    for (int i = tid - kThr; i < zero_count; i += kPlanThreads - kThr) zero_buf[i] = 0;
    return;
  }
  auto barrier = [&]() { asm volatile("bar.sync 1, %0;" ::"n"(kThr) : "memory"); };
  if (tid == 0) plan.hdr[2] = plan.hdr[3] = plan.hdr[4] = 0;
  int e = -1;
  if (tid < P) {
    e = ids[(int64_t)(tid / ids_topk) * ids_ld + (tid % ids_topk)];
    if (expert_map != nullptr) e = (e >= 0 && e < global_E) ? expert_map[e] : -1;
    if (e < 0 || e >= E) e = -1;
    plan.mapped[tid] = e;
    if (e >= 0) s_count[e] = 0;
  }
  __syncwarp();
  barrier();
  int rank = 0;                                // among the pairs of the same expert
  for (int w = 0; w * 32 < P; ++w) {
    if (warp == w) {
      const uint32_t same = __match_any_sync(0xffffffffu, e);
      const int base = e >= 0 ? s_count[e] : 0;
      rank = base + __popc(same & ((1u << lane) - 1));
      __syncwarp();
      if (e >= 0 && (same >> lane) == 1u) s_count[e] = base + __popc(same);        // the highest lane of the group
      __syncwarp();
    }
    barrier();
  }
  // scans over the experts' first pairs: (pairs, experts, passes)
  const int count = e >= 0 ? s_count[e] : 0;
  const bool first = e >= 0 && rank == 0;
  const int sum[3] = {first ? count : 0, first ? 1 : 0, first ? (count + 7) >> 3 : 0};
  int inc[3] = {sum[0], sum[1], sum[2]};
#pragma unroll
  for (int d = 1; d < 32; d <<= 1)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int v = __shfl_up_sync(0xffffffffu, inc[k], d);
      if (lane >= d) inc[k] += v;
    }
  if (lane == 31)
#pragma unroll
    for (int k = 0; k < 3; ++k) s_warp[k][warp] = inc[k];
  __syncwarp();
  barrier();
  int start[3] = {inc[0] - sum[0], inc[1] - sum[1], inc[2] - sum[2]}, total[3] = {0, 0, 0};
#pragma unroll
  for (int w = 0; w < kThr / 32; ++w)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (w < warp) start[k] += s_warp[k][w];
      total[k] += s_warp[k][w];
    }
  if (tid == 0) {
    plan.hdr[0] = total[1];
    plan.hdr[1] = total[2];
  }
  if (first) s_count[e] = start[0] | (start[2] << 16);        // first position in pairs[], first pass
  __syncwarp();
  barrier();
  if (e >= 0) {
    const int pos = (s_count[e] & 0xFFFF) + rank, pass = (s_count[e] >> 16) + (rank >> 3), slot = rank & 7;
    plan.pairs[pos] = tid;
    int* rec = reinterpret_cast<int*>(plan.pass_rec + 2 * pass);        // {expert, tokens, pair0, pair1, pair2, pair3, position, -}
    if (slot < 4) rec[2 + slot] = tid;
    if (slot == 0) {
      rec[0] = e;
      rec[1] = min(8, count - rank);
      rec[6] = pos;
    }
  }
}

// Block 0 builds the plan; the remaining blocks (if any) copy / convert the activation matrix to fp16.
__global__ void __launch_bounds__(kPlanThreads)
    moe_plan_kernel(const int32_t* __restrict__ ids, int P, const int32_t* __restrict__ expert_map, int global_E, int E,
                    Plan plan, const void* __restrict__ conv_src_v, __half* __restrict__ conv_dst,
                    int64_t conv_chunks, int ids_topk, int64_t ids_ld, int64_t conv_row_chunks, int64_t conv_ld_chunks,
                    int* zero_buf, int zero_count, int max_tok, int conv_mode, int conv_block) {
  pdl_wait();                 // the kernel before this one may still be reading the workspace this one rewrites
  pdl_launch_dependents();
  if (blockIdx.x > 0) {
    const uint4* conv_src = reinterpret_cast<const uint4*>(conv_src_v);
    const int64_t stride = (int64_t)(gridDim.x - 1) * kPlanThreads;
    if (conv_mode == kConvBf16) {
      for (int64_t i = (int64_t)(blockIdx.x - 1) * kPlanThreads + threadIdx.x; i < conv_chunks; i += stride) {
        // rows of the source may be strided (conv_ld_chunks 16-byte chunks apart); the copy is dense
        const int64_t row = i / conv_row_chunks, col = i - row * conv_row_chunks;
        const uint4 raw = conv_src[row * conv_ld_chunks + col];
        reinterpret_cast<uint4*>(conv_dst)[i] =
            make_uint4(bf16x2_to_f16x2(raw.x), bf16x2_to_f16x2(raw.y), bf16x2_to_f16x2(raw.z), bf16x2_to_f16x2(raw.w));
      }
    } else {
      // A quad of lanes per group of 32 elements: a 16-byte load each, the 4 x 4 word transpose by shuffles, a 16-byte store each.
      // (A thread per group, 64 bytes in and out, left the copy of 32 tokens to two SMs.)
      const int lane = threadIdx.x & 31;
      for (int64_t i0 = (int64_t)(blockIdx.x - 1) * conv_block; i0 < conv_chunks; i0 += (int64_t)(gridDim.x - 1) * conv_block) {
        for (int j = threadIdx.x; j < conv_block; j += kPlanThreads) {       // whole warps: conv_block is a multiple of 32
          const int64_t i = i0 + j, row = i / conv_row_chunks, col = i - row * conv_row_chunks;
          uint4 v = make_uint4(0, 0, 0, 0);
          if (i < conv_chunks) {
            v = conv_src[row * conv_ld_chunks + col];
            if (conv_mode == kConvBf16Frag) v = make_uint4(bf16x2_to_f16x2(v.x), bf16x2_to_f16x2(v.y), bf16x2_to_f16x2(v.z), bf16x2_to_f16x2(v.w));
          }
          const bool odd = lane & 1, high = lane & 2;
          uint32_t got0 = __shfl_xor_sync(0xffffffffu, odd ? v.x : v.y, 1), got1 = __shfl_xor_sync(0xffffffffu, odd ? v.z : v.w, 1);
          v = odd ? make_uint4(got0, v.y, got1, v.w) : make_uint4(v.x, got0, v.z, got1);
          got0 = __shfl_xor_sync(0xffffffffu, high ? v.x : v.z, 2);
          got1 = __shfl_xor_sync(0xffffffffu, high ? v.y : v.w, 2);
          v = high ? make_uint4(got0, got1, v.z, v.w) : make_uint4(v.x, v.y, got0, got1);
          if (i < conv_chunks) reinterpret_cast<uint4*>(conv_dst)[i] = v;
        }
      }
    }
    return;
  }
  __shared__ int s_count[kPlanMaxExperts];
  __shared__ int s_warp[3][32];
  const int tid = threadIdx.x;
  if (P <= kPlanSmallPairs && max_tok == 8) {
    plan_small(ids, P, expert_map, global_E, E, plan, ids_topk, ids_ld, zero_buf, zero_count, s_count, s_warp);
    return;
  }
  for (int e = tid; e < E; e += kPlanThreads) s_count[e] = 0;
  for (int i = tid; i < zero_count; i += kPlanThreads) zero_buf[i] = 0;   // per-pass counters of the one-launch layer
  if (tid == 0) plan.hdr[2] = plan.hdr[3] = plan.hdr[4] = 0;
  __syncthreads();
  for (int p = tid; p < P; p += kPlanThreads) {
    int e = ids[(int64_t)(p / ids_topk) * ids_ld + (p % ids_topk)];   // ids rows may be strided
    if (expert_map != nullptr) e = (e >= 0 && e < global_E) ? expert_map[e] : -1;
    if (e < 0 || e >= E) e = -1;
    plan.mapped[p] = e;
    if (e >= 0) atomicAdd(&s_count[e], 1);
  }
  __syncthreads();
  // exclusive scans over experts of (pairs, present, passes); each thread owns a contiguous run
  const int per = (E + kPlanThreads - 1) / kPlanThreads;
  const int e0 = tid * per;
  int sum[3] = {0, 0, 0};
  for (int i = 0; i < per; ++i) {
    const int e = e0 + i;
    if (e < E) {
      const int c = s_count[e];
      sum[0] += c;
      sum[1] += c > 0;
      sum[2] += (c + max_tok - 1) / max_tok;
    }
  }
  int inc[3] = {sum[0], sum[1], sum[2]};
  const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int v = __shfl_up_sync(0xffffffffu, inc[k], d);
      if (lane >= d) inc[k] += v;
    }
  if (lane == 31)
#pragma unroll
    for (int k = 0; k < 3; ++k) s_warp[k][warp] = inc[k];
  __syncthreads();
  if (warp == 0) {
    int v[3] = {s_warp[0][lane], s_warp[1][lane], s_warp[2][lane]};
#pragma unroll
    for (int d = 1; d < 32; d <<= 1)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const int x = __shfl_up_sync(0xffffffffu, v[k], d);
        if (lane >= d) v[k] += x;
      }
#pragma unroll
    for (int k = 0; k < 3; ++k) s_warp[k][lane] = v[k];
  }
  __syncthreads();
  int base[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) base[k] = inc[k] - sum[k] + (warp > 0 ? s_warp[k][warp - 1] : 0);
  const int my_pair_base = base[0], my_pass_base = base[2];
  {
    int bc = base[0];
    for (int i = 0; i < per; ++i) {
      const int e = e0 + i;
      if (e < E) {
        const int c = s_count[e];
        s_count[e] = bc;  // becomes the scatter cursor
        bc += c;
      }
    }
  }
  if (tid == kPlanThreads - 1) {
    plan.hdr[0] = base[1] + sum[1];
    plan.hdr[1] = base[2] + sum[2];
  }
  __syncthreads();
  for (int p = tid; p < P; p += kPlanThreads) {
    const int e = plan.mapped[p];
    if (e >= 0) plan.pairs[atomicAdd(&s_count[e], 1)] = p;
  }
  __syncthreads();  // pairs[] (global) written by this block are visible to it after the barrier
  // pass records of the experts this thread owns; after the scatter s_count[e] is the END of e's run
  {
    int start = my_pair_base, pass = my_pass_base;
    for (int i = 0; i < per; ++i) {
      const int e = e0 + i;
      if (e < E) {
        const int end = s_count[e];
        for (int s0 = start; s0 < end; s0 += max_tok) {
          const int nt = min(max_tok, end - s0);
          int pr[4];
#pragma unroll
          for (int t = 0; t < 4; ++t) pr[t] = t < nt ? plan.pairs[s0 + t] : 0;
          // pairs 4.. of an 8-token pass are read from pairs[] (the run of an expert is contiguous there)
          plan.pass_rec[2 * pass] = make_int4(e, nt, pr[0], pr[1]);
          plan.pass_rec[2 * pass + 1] = make_int4(pr[2], pr[3], s0, 0);
          ++pass;
        }
        start = end;
      }
    }
  }
}

// ------------------------------------------------------------------------------------------ tables

__device__ __forceinline__ uint32_t e2m1_to_half_bits(uint32_t nib) {
  const uint32_t c = nib & 7u;
  uint32_t h = (c == 0) ? 0u : (c == 1 ? 0x3800u : 0x3800u + c * 0x200u);
  if (c != 0) h |= (nib & 8u) << 12;
  return h;
}

// Row b (256 bytes) of the table: words 0..31 hold 32 copies of the half2 pair decoded from the
// compressed byte b, words 32..63 hold 32 copies of the two PRMT selectors decoded from the
// metadata byte b.  A lane always reads word `lane` (or 32+lane), i.e. its own bank.
__device__ __forceinline__ void fill_tables(uint32_t* lut, int tid, int nthreads) {
  for (int b = tid; b < 256; b += nthreads) {
    const uint32_t vc = e2m1_to_half_bits(b & 15) | (e2m1_to_half_bits(b >> 4) << 16);
    const uint32_t i0 = b & 3, i1 = (b >> 2) & 3, i2 = (b >> 4) & 3, i3 = (b >> 6) & 3;
    const uint32_t s0 = (2 * i0) | ((2 * i0 + 1) << 4) | ((2 * i1) << 8) | ((2 * i1 + 1) << 12);
    const uint32_t s1 = (2 * i2) | ((2 * i2 + 1) << 4) | ((2 * i3) << 8) | ((2 * i3 + 1) << 12);
    const uint32_t vm = s0 | (s1 << 16);
#pragma unroll 4
    for (int i = 0; i < 32; ++i) {
      const int l = (i + tid) & 31;  // rotate so that the 32 threads of a warp hit 32 banks
      lut[b * 64 + l] = vc;
      lut[b * 64 + 32 + l] = vm;
    }
  }
}

// ------------------------------------------------------------------------------------------ GEMV

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async8(void* smem_dst, const void* gmem_src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(gmem_src) : "memory");
}
// COLS bytes (16 or 8) of one weight row
template <int COLS>
__device__ __forceinline__ void cp_async_cols(void* smem_dst, const void* gmem_src) {
  if (COLS == 16) cp_async16(smem_dst, gmem_src);
  else cp_async8(smem_dst, gmem_src);
}
__device__ __forceinline__ uint32_t lds32(const unsigned char* p) { return *reinterpret_cast<const uint32_t*>(p); }

// One scale block (16 k) x 16 columns for T tokens.  v[] = 4 compressed rows, 2 metadata rows,
// 1 (or 2) scale rows; a[t] = the 16 activations of token t as 8 half2.
template <int T, int COLS, bool kScale8>
__device__ __forceinline__ void compute_block(const uint4 (&v)[8], const uint4 (&a)[T][2], const unsigned char* lut,
                                              uint32_t lane4, float (&acc)[T][COLS]) {
  // PRMT selectors: (table row = byte j of the word) << 8 | lane*4
  constexpr uint32_t kIdx[4] = {0x5504u, 0x5514u, 0x5524u, 0x5534u};
  // PRMT selectors: bytes (j, j+1) of the scale word to the high bytes of two halves
  constexpr uint32_t kSc[2] = {0x1404u, 0x3424u};
#pragma unroll
  for (int q = 0; q < COLS / 4; ++q) {
    const uint32_t c0 = word_of(v[0], q), c1 = word_of(v[1], q), c2 = word_of(v[2], q), c3 = word_of(v[3], q);
    const uint32_t m0 = word_of(v[4], q), m1 = word_of(v[5], q);
    const uint32_t s0 = word_of(v[6], q) & 0x7F7F7F7Fu;
    const uint32_t s1 = kScale8 ? (word_of(v[7], q) & 0x7F7F7F7Fu) : 0u;
#pragma unroll
    for (int jp = 0; jp < 2; ++jp) {
      // e4m3 bits moved into a half give scale * 2^-8; the 2^8 is folded into the final multiplier
      const float2 sc0 = __half22float2(as_h2(prmt(s0, 0u, kSc[jp]) >> 1));
      float2 sc1 = make_float2(0.f, 0.f);
      if (kScale8) sc1 = __half22float2(as_h2(prmt(s1, 0u, kSc[jp]) >> 1));
#pragma unroll
      for (int jj = 0; jj < 2; ++jj) {
        const int j = jp * 2 + jj;
        const int col = q * 4 + j;
        const __half2 w0 = as_h2(lds32(lut + prmt(c0, lane4, kIdx[j])));
        const __half2 w1 = as_h2(lds32(lut + prmt(c1, lane4, kIdx[j])));
        const __half2 w2 = as_h2(lds32(lut + prmt(c2, lane4, kIdx[j])));
        const __half2 w3 = as_h2(lds32(lut + prmt(c3, lane4, kIdx[j])));
        const uint32_t sel01 = lds32(lut + 128 + prmt(m0, lane4, kIdx[j]));
        const uint32_t sel23 = lds32(lut + 128 + prmt(m1, lane4, kIdx[j]));
        const uint32_t sel1 = sel01 >> 16, sel3 = sel23 >> 16;
        const float f0 = jj == 0 ? sc0.x : sc0.y;
        const float f1 = jj == 0 ? sc1.x : sc1.y;
#pragma unroll
        for (int t = 0; t < T; ++t) {
          __half2 p = __hmul2(w0, as_h2(prmt(a[t][0].x, a[t][0].y, sel01)));
          p = __hfma2(w1, as_h2(prmt(a[t][0].z, a[t][0].w, sel1)), p);
          if (kScale8) {
            __half2 r = __hmul2(w2, as_h2(prmt(a[t][1].x, a[t][1].y, sel23)));
            r = __hfma2(w3, as_h2(prmt(a[t][1].z, a[t][1].w, sel3)), r);
            acc[t][col] = fmaf(__half2float(__hadd(__low2half(p), __high2half(p))), f0, acc[t][col]);
            acc[t][col] = fmaf(__half2float(__hadd(__low2half(r), __high2half(r))), f1, acc[t][col]);
          } else {
            p = __hfma2(w2, as_h2(prmt(a[t][1].x, a[t][1].y, sel23)), p);
            p = __hfma2(w3, as_h2(prmt(a[t][1].z, a[t][1].w, sel3)), p);
            acc[t][col] = fmaf(__half2float(__hadd(__low2half(p), __high2half(p))), f0, acc[t][col]);
          }
        }
      }
    }
  }
}

__device__ __forceinline__ void store_out(void* out, int dtype, int64_t idx, float v) {
  if (dtype == B200FP4_DTYPE_F16) reinterpret_cast<__half*>(out)[idx] = __float2half_rn(v);
  else if (dtype == B200FP4_DTYPE_BF16) reinterpret_cast<__nv_bfloat16*>(out)[idx] = __float2bfloat16_rn(v);
  else reinterpret_cast<float*>(out)[idx] = v;
}

struct Rec {
  int e, nt;
  int p0, p1, p2, p3;
  __device__ __forceinline__ int pair(int t) const { return t == 0 ? p0 : (t == 1 ? p1 : (t == 2 ? p2 : p3)); }
};
__device__ __forceinline__ Rec load_rec(const int4* recs, int pass) {
  const int4 x = recs[2 * pass], y = recs[2 * pass + 1];
  Rec r;
  r.e = x.x; r.nt = x.y; r.p0 = x.z; r.p1 = x.w; r.p2 = y.x; r.p3 = y.y;
  return r;
}
__device__ __forceinline__ Rec empty_rec() {
  Rec r;
  r.e = -1; r.nt = 0; r.p0 = r.p1 = r.p2 = r.p3 = 0;
  return r;
}

// NT      threads per block: 256 with COLS = 16 columns per thread, or 512 with COLS = 8 (twice the
//         warps per SM for latency hiding, half the accumulators per thread)
// CG      column groups per slab: slab = COLS*CG columns, NT/CG K-slices
// S       cp.async ring stages; every thread must own at least S-1 scale blocks per item
// kScale8 one scale per 8 k instead of per 16 k
// kSilu   slab = CG*8 gate columns + the matching CG*8 up columns; epilogue writes SiLU(gate)*up
template <int NT, int COLS, int CG, int S, bool kScale8, bool kSilu>
__global__ void __launch_bounds__(NT, 1) sparse_gemv_kernel(const GemvArgs g) {
  constexpr int kThreads = NT;
  constexpr int kWarps = NT / 32;
  constexpr int KS = kThreads / CG;
  constexpr int SLAB = CG * COLS;
  constexpr int NV = kScale8 ? 8 : 7;
  using Vec = typename std::conditional<COLS == 16, uint4, uint2>::type;   // COLS bytes of one weight row
  extern __shared__ __align__(16) unsigned char smem[];
  uint32_t* lut_w = reinterpret_cast<uint32_t*>(smem);
  Vec* ring = reinterpret_cast<Vec*>(smem + kLutBytes);                          // [S][NV][NT]
  float* red = reinterpret_cast<float*>(ring + S * NV * kThreads);               // [kWarps][kMaxTok][SLAB]
  __half* sA = reinterpret_cast<__half*>(red + kWarps * kMaxTok * SLAB);         // [2][kMaxTok][K]

  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int cg = lane % CG, ksub = lane / CG;
  const int kslice = warp * (32 / CG) + ksub;
  const uint32_t lane4 = (uint32_t)lane * 4u;
  const int K = g.K, KB = K >> 4;
  const int nblk = (KB - kslice + KS - 1) / KS;   // scale blocks this thread owns in every item (>= S-1)
  const int grid = gridDim.x;
  fill_tables(lut_w, tid, kThreads);

  const int n_items = g.plan.hdr[1] * g.n_slabs;
  int item = blockIdx.x;
  if (item >= n_items) return;
  Rec rc = load_rec(g.plan.pass_rec, item / g.n_slabs);
  Rec rn = (item + grid < n_items) ? load_rec(g.plan.pass_rec, (item + grid) / g.n_slabs) : empty_rec();

  // this thread's share of the activation rows of a pass -> sA[buf]
  const int chunks = K >> 3;
  auto issue_A = [&](const Rec& r, int buf) {
    for (int i = tid; i < r.nt * chunks; i += kThreads) {
      const int t = i / chunks, ch = i - t * chunks;
      const int64_t row = r.pair(t) / g.a_div;
      cp_async16(sA + ((size_t)(buf * kMaxTok + t) * K + ch * 8), g.A + row * g.lda + ch * 8);
    }
  };

  // ---- weight fetch stream: runs S-1 blocks ahead of the compute and crosses item boundaries
  int f_item = item, f_j = 0, f_slot = 0;
  const uint8_t *f_comp = nullptr, *f_meta = nullptr, *f_scale = nullptr;
  bool f_ok = false;
  auto fetch_next = [&](const Rec& cur, const Rec& nxt) {
    if (f_item < n_items) {
      if (f_j == 0) {
        const int e = (f_item == item) ? cur.e : nxt.e;
        const int slab = f_item % g.n_slabs;
        int col0;
        if (kSilu) col0 = (cg < CG / 2) ? slab * (SLAB / 2) + cg * COLS : g.inter + slab * (SLAB / 2) + (cg - CG / 2) * COLS;
        else col0 = slab * SLAB + cg * COLS;
        f_ok = kSilu ? ((cg < CG / 2 ? col0 : col0 - g.inter) < g.inter) : (col0 < g.N);
        f_comp = g.w.comp + (int64_t)e * g.w.comp_e + col0;
        f_meta = g.w.meta + (int64_t)e * g.w.meta_e + col0;
        f_scale = g.w.scale + (int64_t)e * g.w.scale_e + col0;
      }
      if (f_ok) {
        const int kb = kslice + KS * f_j;
        Vec* dst = ring + (size_t)f_slot * NV * kThreads + tid;
        const uint8_t* c0 = f_comp + (int64_t)(2 * kb) * g.w.comp_pair;
        cp_async_cols<COLS>(dst, c0);
        cp_async_cols<COLS>(dst + kThreads, c0 + g.w.comp_odd);
        cp_async_cols<COLS>(dst + 2 * kThreads, c0 + g.w.comp_pair);
        cp_async_cols<COLS>(dst + 3 * kThreads, c0 + g.w.comp_pair + g.w.comp_odd);
        const uint8_t* m0 = f_meta + (int64_t)(2 * kb) * g.w.meta_row;
        cp_async_cols<COLS>(dst + 4 * kThreads, m0);
        cp_async_cols<COLS>(dst + 5 * kThreads, m0 + g.w.meta_row);
        if (kScale8) {
          const uint8_t* s0 = f_scale + (int64_t)(2 * kb) * g.w.scale_row;
          cp_async_cols<COLS>(dst + 6 * kThreads, s0);
          cp_async_cols<COLS>(dst + 7 * kThreads, s0 + g.w.scale_row);
        } else {
          cp_async_cols<COLS>(dst + 6 * kThreads, f_scale + (int64_t)kb * g.w.scale_row);
        }
      }
      if (++f_j == nblk) {
        f_j = 0;
        f_item += grid;
      }
    }
    cp_async_commit();
    f_slot = (f_slot + 1 == S) ? 0 : f_slot + 1;
  };

  // prologue: activations of the first item, then S-1 weight blocks
  issue_A(rc, 0);
  cp_async_commit();
#pragma unroll
  for (int s = 0; s < S - 1; ++s) fetch_next(rc, rn);

  int c_slot = 0, abuf = 0;
  for (; item < n_items; item += grid) {
    const int slab = item % g.n_slabs;
    // record of the item after next; activations of the next item ride on the next weight group
    Rec rnn = (item + 2 * grid < n_items) ? load_rec(g.plan.pass_rec, (item + 2 * grid) / g.n_slabs) : empty_rec();
    const float gmul = g.w.g[rc.e] * 256.0f;
    cp_async_wait<S - 2>();   // oldest group: first weight block of this item and (older) its activations
    __syncthreads();          // sA[abuf] complete for all threads; red and sA[abuf^1] free
    issue_A(rn, abuf ^ 1);

    float accs[kMaxTok][COLS];
    auto run = [&](auto tconst) {
      constexpr int T = decltype(tconst)::value;
      float acc[T][COLS];
#pragma unroll
      for (int t = 0; t < T; ++t)
#pragma unroll
        for (int c = 0; c < COLS; ++c) acc[t][c] = 0.f;
      for (int j = 0; j < nblk; ++j) {
        cp_async_wait<S - 2>();
        uint4 v[8];
        const Vec* src = ring + (size_t)c_slot * NV * kThreads + tid;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          const Vec x = src[i * kThreads];
          v[i].x = x.x;
          v[i].y = x.y;
          if (COLS == 16) {
            v[i].z = reinterpret_cast<const uint32_t*>(&x)[COLS == 16 ? 2 : 0];
            v[i].w = reinterpret_cast<const uint32_t*>(&x)[COLS == 16 ? 3 : 0];
          } else {
            v[i].z = v[i].w = 0u;
          }
        }
        if (!kScale8) v[7] = make_uint4(0, 0, 0, 0);
        fetch_next(rc, rn);
        const int kb = kslice + KS * j;
        uint4 a[T][2];
#pragma unroll
        for (int t = 0; t < T; ++t) {
          const uint4* pa = reinterpret_cast<const uint4*>(sA + ((size_t)(abuf * kMaxTok + t) * K + (size_t)kb * 16));
          a[t][0] = pa[0];
          a[t][1] = pa[1];
        }
        compute_block<T, COLS, kScale8>(v, a, smem, lane4, acc);
        c_slot = (c_slot + 1 == S) ? 0 : c_slot + 1;
      }
      // K reduction: the K-slices of a warp through shuffles, then the warps through shared memory
#pragma unroll
      for (int t = 0; t < T; ++t)
#pragma unroll
        for (int c = 0; c < COLS; ++c) {
          float x = acc[t][c];
#pragma unroll
          for (int d = CG; d < 32; d <<= 1) x += __shfl_xor_sync(0xffffffffu, x, d);
          accs[t][c] = x;
        }
      if (ksub == 0) {
#pragma unroll
        for (int t = 0; t < T; ++t) {
          float4* dst = reinterpret_cast<float4*>(red + ((size_t)warp * kMaxTok + t) * SLAB + cg * COLS);
#pragma unroll
          for (int c = 0; c < COLS / 4; ++c)
            dst[c] = make_float4(accs[t][4 * c], accs[t][4 * c + 1], accs[t][4 * c + 2], accs[t][4 * c + 3]);
        }
      }
    };
    if (rc.nt == 1) run(std::integral_constant<int, 1>{});
    else if (rc.nt == 2) run(std::integral_constant<int, 2>{});
    else if (rc.nt == 3) run(std::integral_constant<int, 3>{});
    else run(std::integral_constant<int, 4>{});
    __syncthreads();
    // epilogue: sum the warps, apply the expert's global scale, write
    if (kSilu) {
      constexpr int HALF = SLAB / 2;
      for (int i = tid; i < rc.nt * HALF; i += kThreads) {
        const int t = i / HALF, j = i - t * HALF;
        const int n = slab * HALF + j;
        if (n < g.inter) {
          float gate = 0.f, up = 0.f;
#pragma unroll
          for (int w = 0; w < kWarps; ++w) {
            gate += red[((size_t)w * kMaxTok + t) * SLAB + j];
            up += red[((size_t)w * kMaxTok + t) * SLAB + HALF + j];
          }
          gate *= gmul;
          up *= gmul;
          const float act = gate / (1.0f + __expf(-gate)) * up;
          store_out(g.out, g.out_dtype, (int64_t)rc.pair(t) * g.ldo + n, act);
        }
      }
    } else {
      for (int i = tid; i < rc.nt * SLAB; i += kThreads) {
        const int t = i / SLAB, j = i - t * SLAB;
        const int n = slab * SLAB + j;
        if (n < g.N) {
          float x = 0.f;
#pragma unroll
          for (int w = 0; w < kWarps; ++w) x += red[((size_t)w * kMaxTok + t) * SLAB + j];
          store_out(g.out, g.out_dtype, (int64_t)rc.pair(t) * g.ldo + n, x * gmul);
        }
      }
    }
    rc = rn;
    rn = rnn;
    abuf ^= 1;
  }
  cp_async_wait<0>();
}

// Rows of pairs whose expert is not local are never touched by the GEMV; this writes zeros there.
__global__ void zero_unmapped_rows_kernel(const int* __restrict__ mapped, int P, void* out, int out_dtype, int64_t ldo,
                                          int N) {
  const int p = blockIdx.x;
  if (p >= P || mapped[p] >= 0) return;
  for (int n = threadIdx.x; n < N; n += blockDim.x) store_out(out, out_dtype, (int64_t)p * ldo + n, 0.f);
}

// four neighbouring results
__device__ __forceinline__ void store_out4(void* out, int dtype, int64_t idx, const float4& v) {
  if (dtype == B200FP4_DTYPE_F32) {
    *reinterpret_cast<float4*>(reinterpret_cast<float*>(out) + idx) = v;
  } else if (dtype == B200FP4_DTYPE_F16) {
    const __half2 lo = __floats2half2_rn(v.x, v.y), hi = __floats2half2_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(out) + idx) =
        make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
  } else {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(out) + idx) =
        make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
  }
}

// Pass record of the tensor-core kernel: up to TM (4 or 8) pairs.
template <int TM>
struct RecT {
  int e, nt;
  int p[TM];
  __device__ __forceinline__ int pair(int t) const {
    int v = p[0];
#pragma unroll
    for (int i = 1; i < TM; ++i) v = (t == i) ? p[i] : v;
    return v;
  }
};
template <int TM>
__device__ __forceinline__ RecT<TM> load_rec_t(const Plan& plan, int pass) {
  const int4 x = plan.pass_rec[2 * pass], y = plan.pass_rec[2 * pass + 1];
  RecT<TM> r;
  r.e = x.x; r.nt = x.y; r.p[0] = x.z; r.p[1] = x.w; r.p[2] = y.x; r.p[3] = y.y;
  if (TM == 8) {
#pragma unroll
    for (int i = 4; i < TM; ++i) r.p[i] = (i < r.nt) ? plan.pairs[y.z + i] : 0;
  }
  return r;
}
template <int TM>
__device__ __forceinline__ RecT<TM> empty_rec_t() {
  RecT<TM> r;
  r.e = -1; r.nt = 0;
#pragma unroll
  for (int i = 0; i < TM; ++i) r.p[i] = 0;
  return r;
}

// ------------------------------------------------------------------------------------------ tensor-core GEMV
//
// Same work items as sparse_gemv_kernel, but the 2:4 gather and the multiply-accumulate run on the
// tensor cores: the weights are the sparse A operand of mma.sp m16n8k32 (f16, fp32 accumulate), the
// reference's metadata bytes are -- after one byte permute -- the instruction's metadata operand, and
// the (up to four, or eight) tokens of the pass are columns of B.  What is left for the CUDA cores is the
// E2M1 -> half2 decode (cvt.rn.f16x2.e2m1x2 straight from a byte of the loaded word), the E4M3 ->
// half2 decode of the block scales (cvt.rn.f16x2.e4m3x2) and one half2 multiply per pair of weights
// (E2M1 x E4M3 is exact in fp16).
//
// Requires every 4-group's two indices in increasing order (the instruction's rule), which is how
// the reference's converter writes them (sparse_v7_moe_patch.py:59-60); callers promise it.
//
// A block is 16 warps.  An item is (pass, slab of 128*CG columns); warp w owns column group w % CG
// and K-slice w / CG and walks its K-slice in steps of 32 k.  One step of one warp reads 8 compressed
// rows, 4 metadata rows and 2 scale rows of 128 columns (1792 bytes) from a private cp.async ring
// that keeps running across items, and issues 8 mma.sp (16 columns x 32 k each):
//   * quad q = lane / 4 owns columns 16q..16q+15 of the warp's 128; mma j takes columns 2h, 2h+1 of
//     every quad (h = 4*(j%2) + j/2) as its rows q and q+8;
//   * lane t = lane % 4 of the quad reads compressed rows t and t+4 (the instruction's 4-groups t and
//     t+4), so byte 2h (2h+1) of those two 16-byte vectors decodes to the fragment registers of row q
//     (q+8) -- no shuffles;
//   * metadata: for mma j the lanes with t/2 == j%2 supply it; their register is [row q | row q+8] x
//     [metadata rows 2(t%2), 2(t%2)+1], i.e. bytes (2h, 2h+1) of two 8-byte loads interleaved by PRMT.
constexpr int kMmaThreads = 512;
constexpr int kMmaWarps = 16;
constexpr int kMmaStageBytes = 1792;
constexpr int kMmaRedBytes = kMmaWarps * 128 * 4 * 4;   // K-slice partial sums [warp][column][token] fp32

// One projection over all items of this block.
// TM = tokens per pass (4 or 8; the instruction's B operand has 8 columns either way, but the
// activation buffers and the partial-sum scratch double with 8).
template <int CG, int S, bool kSilu, int TM>
__device__ __forceinline__ void gemv_mma_phase(const GemvArgs& g, unsigned char* smem) {
  using Rec = RecT<TM>;
  constexpr int KSL = kMmaWarps / CG;          // K-slices per item
  constexpr int VCOLS = 128 * CG;              // columns of a slab (SiLU: 64*CG gate + 64*CG up)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int q = lane >> 2, t = lane & 3;
  const int cgw = warp % CG, ks = warp / CG;
  const int K = g.K;
  const int nstep = K / (32 * KSL);
  const int grid = gridDim.x;

  // ---- shared memory map (shared-window addresses)
  //   activations of the current and the next pass [2][TM][K + 8] fp16 | partial sums (one block of
  //   kMmaRedBytes per four tokens) | 16 rings of S stages
  const uint32_t a_pitch = 2u * (uint32_t)K + 16u;
  const uint32_t sa = (shared_addr(smem) + 1023u) & ~1023u;
  const uint32_t red = sa + ((2u * TM * a_pitch + 1023u) & ~1023u);
  const uint32_t ring_bytes = S * kMmaStageBytes;
  const uint32_t ring = red + (TM / 4) * kMmaRedBytes + (uint32_t)warp * ring_bytes;
  const uint32_t ring_end = ring + ring_bytes;

  // ---- items of this block: blockIdx.x, + grid, ...
  const int n_slabs = g.n_slabs;
  const int n_items = g.plan.hdr[1] * n_slabs;
  const int my_items = (int)blockIdx.x < n_items ? (n_items - 1 - (int)blockIdx.x) / grid + 1 : 0;
  if (my_items == 0) return;
  auto pass_of = [&](int i) { return ((int)blockIdx.x + i * grid) / n_slabs; };
  Rec rc = load_rec_t<TM>(g.plan, pass_of(0));
  Rec rn = my_items > 1 ? load_rec_t<TM>(g.plan, pass_of(1)) : empty_rec_t<TM>();
  int e_nn = my_items > 2 ? g.plan.pass_rec[2 * pass_of(2)].x : -1;

  const int chunks = K >> 3;
  auto issue_A = [&](const Rec& r, int buf) {
#pragma unroll
    for (int tk = 0; tk < TM; ++tk)
      if (tk < r.nt) {
        const uint32_t pr = (uint32_t)r.p[tk];
        const int64_t row = g.a_magic ? (int64_t)__umulhi(pr, g.a_magic) : (int64_t)pr;
        const __half* src = g.A + row * g.lda;
        const uint32_t dst = sa + (uint32_t)(buf * TM + tk) * a_pitch;
        for (int ch = tid; ch < chunks; ch += kMmaThreads) cp_async16_s(dst + (uint32_t)ch * 16u, src + ch * 8);
      }
  };

  // ---- weight fetch stream of this warp: lane = (row fr, 16-byte chunk fc) of every tensor's tile.
  // It runs S-1 stages ahead of the compute and crosses item boundaries (at most two items ahead).
  const int fr = lane >> 3, fc = lane & 7;
  const int64_t comp_step = 4 * g.w.comp_pair * KSL, meta_step = 4 * g.w.meta_row * KSL, scale_step = 2 * g.w.scale_row * KSL;
  const int64_t comp_row4 = 2 * g.w.comp_pair;
  const int64_t lane_comp = (int64_t)(4 * ks + (fr >> 1)) * g.w.comp_pair + (fr & 1) * g.w.comp_odd;
  const int64_t lane_meta = (int64_t)(4 * ks + fr) * g.w.meta_row;
  const int64_t lane_scale = (int64_t)(2 * ks + fr) * g.w.scale_row;
  const int lane_v = cgw * 128 + fc * 16;   // virtual column of this lane's chunk in the slab
  int i_cur = 0;                            // ordinal of the item being computed
  int f_i = 0, f_j = 0;
  uint32_t f_dst = ring + (uint32_t)lane * 16u;
  const uint8_t *f_comp = nullptr, *f_meta = nullptr, *f_scale = nullptr;
  auto fetch_next = [&]() {
    if (f_i < my_items) {
      if (f_j == 0) {
        const int rel = f_i - i_cur;
        const int e = rel == 0 ? rc.e : (rel == 1 ? rn.e : e_nn);
        const int slab = ((int)blockIdx.x + f_i * grid) % n_slabs;
        int col;
        if (kSilu) col = lane_v < 64 * CG ? slab * (64 * CG) + lane_v : g.inter + slab * (64 * CG) + (lane_v - 64 * CG);
        else col = slab * VCOLS + lane_v;
        f_comp = g.w.comp + ((int64_t)e * g.w.comp_e + col + lane_comp);
        f_meta = g.w.meta + ((int64_t)e * g.w.meta_e + col + lane_meta);
        f_scale = g.w.scale + ((int64_t)e * g.w.scale_e + col + lane_scale);
      }
      cp_async16_s(f_dst, f_comp);
      cp_async16_s(f_dst + 512u, f_comp + comp_row4);
      cp_async16_s(f_dst + 1024u, f_meta);
      if (lane < 16) cp_async16_s(f_dst + 1536u, f_scale);
      f_comp += comp_step;
      f_meta += meta_step;
      f_scale += scale_step;
      if (++f_j == nstep) {
        f_j = 0;
        ++f_i;
      }
    }
    cp_async_commit();
    f_dst += kMmaStageBytes;
    if (f_dst >= ring_end) f_dst -= ring_bytes;
  };

  issue_A(rc, 0);
  cp_async_commit();
#pragma unroll
  for (int s = 0; s < S - 1; ++s) fetch_next();

  // lane-constant pieces of the addresses used in a step
  const uint32_t off_comp = (uint32_t)t * 128u + (uint32_t)q * 16u;
  const uint32_t off_meta = 1024u + (uint32_t)(2 * (t & 1)) * 128u + (uint32_t)q * 16u + (uint32_t)(t >> 1) * 8u;
  const uint32_t off_scale = 1536u + (uint32_t)q * 16u;
  // B column q = token q (with four tokens per pass columns 4..7 repeat them; their results are never read),
  // k = 32*ks + 2t (+8i)
  const uint32_t off_b = (uint32_t)(TM == 8 ? q : (q & 3)) * a_pitch + (uint32_t)t * 4u + (uint32_t)ks * 64u;
  // scratch [warp][column 0..127][token 0..3]; the 16-byte token groups of a column are XOR-swizzled
  // by the column's quad so that neither side has bank conflicts
  // (tokens 4..7 of an 8-token pass, held by lanes t = 2, 3, go to a second block of the same shape)
  const uint32_t red_w = red + (uint32_t)(t >> 1) * kMmaRedBytes + (uint32_t)warp * 2048u + (uint32_t)q * 256u +
                         8u * (uint32_t)(t & 1) + 16u * (uint32_t)((q ^ ((cgw & 1) << 2)) & 7);

  uint32_t c_st = ring;
  int abuf = 0;
  for (; i_cur < my_items; ++i_cur) {
    const int slab = ((int)blockIdx.x + i_cur * grid) % n_slabs;
    Rec rnn = i_cur + 2 < my_items ? load_rec_t<TM>(g.plan, pass_of(i_cur + 2)) : empty_rec_t<TM>();
    const int e_n3 = i_cur + 3 < my_items ? g.plan.pass_rec[2 * pass_of(i_cur + 3)].x : -1;
    const float gmul = g.w.g[rc.e];
    // the group that carried this pass's activations is followed by nstep - 1 newer ones
    if (nstep >= S - 1) cp_async_wait<S - 2>();
    else if (nstep == 2) cp_async_wait<1>();
    else cp_async_wait<(S > 3 ? 2 : 1)>();
    __syncthreads();   // activations of this pass complete for all threads; scratch and the other buffer free
    issue_A(rn, abuf ^ 1);   // rides on the next committed weight stage

    float acc[8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[j][k] = 0.f;
    uint32_t ab = sa + (uint32_t)abuf * TM * a_pitch + off_b;

    for (int js = 0; js < nstep; ++js) {
      cp_async_wait<S - 2>();
      __syncwarp();
      const uint32_t st = c_st;
      const uint4 v0 = lds128_at(st + off_comp), v1 = lds128_at(st + off_comp + 512u);
      const uint2 m0 = lds64_at(st + off_meta), m1 = lds64_at(st + off_meta + 128u);
      const uint4 s0 = lds128_at(st + off_scale), s1 = lds128_at(st + off_scale + 128u);
      uint32_t b[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) b[k] = lds32_at(ab + 16u * k);
      ab += 64u * KSL;
      c_st += kMmaStageBytes;
      if (c_st >= ring_end) c_st -= ring_bytes;
      fetch_next();   // into the slot read in the previous step (all lanes are past this step's __syncwarp)
      uint32_t em[4];
      em[0] = prmt(m0.x, m1.x, 0x5140u);
      em[1] = prmt(m0.x, m1.x, 0x7362u);
      em[2] = prmt(m0.y, m1.y, 0x5140u);
      em[3] = prmt(m0.y, m1.y, 0x7362u);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        // mma j: columns 2h, 2h+1 of the quad = bytes (2hf, 2hf+1) of word wi of every loaded vector
        constexpr int kH[8] = {0, 4, 1, 5, 2, 6, 3, 7};
        const int h = kH[j];
        const int wi = h >> 1, hf = h & 1;
        const uint32_t c0 = word_of(v0, wi), c1 = word_of(v1, wi);
        const __half2 sc0 = hf ? e4m3x2_to_h2<1>(word_of(s0, wi)) : e4m3x2_to_h2<0>(word_of(s0, wi));
        const __half2 sc1 = hf ? e4m3x2_to_h2<1>(word_of(s1, wi)) : e4m3x2_to_h2<0>(word_of(s1, wi));
        const __half2 a0 = __hmul2(hf ? e2m1x2_to_h2<2>(c0) : e2m1x2_to_h2<0>(c0), __low2half2(sc0));
        const __half2 a1 = __hmul2(hf ? e2m1x2_to_h2<3>(c0) : e2m1x2_to_h2<1>(c0), __high2half2(sc0));
        const __half2 a2 = __hmul2(hf ? e2m1x2_to_h2<2>(c1) : e2m1x2_to_h2<0>(c1), __low2half2(sc1));
        const __half2 a3 = __hmul2(hf ? e2m1x2_to_h2<3>(c1) : e2m1x2_to_h2<1>(c1), __high2half2(sc1));
        if ((j & 1) == 0)
          mma_sp_m16n8k32<0>(acc[j], *reinterpret_cast<const uint32_t*>(&a0), *reinterpret_cast<const uint32_t*>(&a1),
                             *reinterpret_cast<const uint32_t*>(&a2), *reinterpret_cast<const uint32_t*>(&a3), b, em[j >> 1]);
        else
          mma_sp_m16n8k32<1>(acc[j], *reinterpret_cast<const uint32_t*>(&a0), *reinterpret_cast<const uint32_t*>(&a1),
                             *reinterpret_cast<const uint32_t*>(&a2), *reinterpret_cast<const uint32_t*>(&a3), b, em[j >> 1]);
      }
    }

    // partial sums of this K-slice -> scratch
    if (2 * t < rc.nt) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        constexpr int kH[8] = {0, 4, 1, 5, 2, 6, 3, 7};
        const uint32_t c0 = 2u * kH[j], c1 = 2u * kH[j] + 1u;   // columns of the quad: rows q and q+8 of mma j
        sts64f_at((red_w ^ ((c0 & 7u) << 4)) + (c0 >> 3) * 128u, acc[j][0], acc[j][1]);
        sts64f_at((red_w ^ ((c1 & 7u) << 4)) + (c1 >> 3) * 128u, acc[j][2], acc[j][3]);
      }
    }
    __syncthreads();
    // epilogue, spread over all warps: one (column, token) sum per lane and round.  The warp of
    // K-slice s and column group cw is s * CG + cw.
    auto slice_sum = [&](int v, int tok) {
      const int cw = v >> 7, col = v & 127;
      const uint32_t a = red + (uint32_t)(tok >> 2) * kMmaRedBytes + (uint32_t)cw * 2048u +
                         (((uint32_t)col * 16u) ^ ((uint32_t)(((col >> 4) ^ ((cw & 1) << 2)) & 7) << 4)) + (uint32_t)(tok & 3) * 4u;
      float sum = 0.f;
#pragma unroll
      for (int s = 0; s < KSL; ++s) sum += __uint_as_float(lds32_at(a + (uint32_t)(s * CG) * 2048u));
      return sum;
    };
    if (kSilu) {
#pragma unroll
      for (int r = 0; r < CG * (TM / 4); ++r) {
        const int idx = (r % CG) * 256 + warp * 16 + (lane & 15);
        const int col_g = idx >> 2, tok = (idx & 3) + 4 * (r / CG);
        const float sum = slice_sum(col_g + (lane >> 4) * (64 * CG), tok);
        const float other = __shfl_down_sync(0xffffffffu, sum, 16);
        if (lane < 16 && tok < rc.nt) {
          const float gate = sum * gmul, up = other * gmul;
          store_out(g.out, g.out_dtype, (int64_t)rc.pair(tok) * g.ldo + slab * (64 * CG) + col_g,
                    gate / (1.0f + __expf(-gate)) * up);
        }
      }
    } else {
#pragma unroll
      for (int r = 0; r < CG * (TM / 4); ++r) {
        const int x = (r % CG) * 512 + tid;
        const int v = x >> 2, tok = (x & 3) + 4 * (r / CG);
        const float sum = slice_sum(v, tok);
        if (tok < rc.nt) store_out(g.out, g.out_dtype, (int64_t)rc.pair(tok) * g.ldo + slab * VCOLS + v, sum * gmul);
      }
    }
    rc = rn;
    rn = rnn;
    e_nn = e_n3;
    abuf ^= 1;
  }
  cp_async_wait<0>();
}

// Programmatic dependent launch: the GEMV and reduce kernels of a layer are launched with the stream-serialization
// attribute, so their blocks may become resident while the kernel before them drains; pdl_wait() returns once that
// kernel has completed and its writes are visible (at once when the launch carried no such attribute).


template <int CG, int S, bool kSilu, int TM>
__global__ void __launch_bounds__(kMmaThreads, 1) sparse_gemv_mma_kernel(const GemvArgs g) {
  extern __shared__ __align__(16) unsigned char smem[];
  pdl_wait();
  pdl_launch_dependents();
  gemv_mma_phase<CG, S, kSilu, TM>(g, smem);
}

// ------------------------------------------------------------------------------------------ warp-scheduled tensor-core GEMV
//
// The same arithmetic as gemv_mma_phase (mma.sp m16n8k32, hardware E2M1 / E4M3 decode), organised so that a warp
// never has to meet another warp:
//   * a work item is (pass of up to eight tokens, group of 128 output columns) over the WHOLE K, owned by one warp:
//     no K-slices, so no partial sums in shared memory, no block-wide barrier and no block-wide epilogue (in the layer's
//     one launch two or four warps share an item where items are few, see KS below);
//   * warps take items from a global counter (atomicAdd by lane 0), always holding the next item while they
//     compute the current one, so the tail of the launch is at most one item long whatever the routing;
//   * the activations are not staged per block: the plan kernel (or the gate_up epilogue) leaves them in
//     "fragment order" (see kConv*), and each lane copies the 16 bytes that are its own B-operand registers for a
//     k-step asynchronously into its ring stage, next to the weights of that step;
//   * a ring stage is one 32-wide k-step: 8 compressed rows, 4 metadata rows and 2 scale rows of 128 columns
//     (1792 bytes) + 512 bytes of B fragments.  kS stages per warp (four or eight); the copy for step j+kS is issued into
//     the slot of step j as soon as step j's shared-memory reads are done, so that kS steps are in flight per warp and the
//     slot of every step is a compile-time constant in the loop unrolled by kS (a warp's share of K is whole turns).  The
//     stream runs across item boundaries.
//   * 16-byte chunks are XOR-swizzled inside the compressed and metadata rows so that the fragment loads
//     (rows t and t+4 for lane t of a quad; metadata rows 2(t%2), 2(t%2)+1) touch every bank once.
// Epilogue from registers: the lane that holds 16 consecutive columns of a token writes them with 16-byte stores;
// with SiLU the warp's 128 columns are 64 gate + the matching 64 up columns, the two halves of the warp swap one
// token's values through shuffles, and SiLU(gate)*up leaves in fragment order for the down projection.
// Which blocks and rings: see launch_fused_ws for the layer; a stand-alone projection takes 8 warps x 8 stages where K is a
// multiple of 256, else 16 warps x 4 stages.
// One projection for this warp: the items [base, base + passes * groups) of the claim sequence that `counter` hands out.
// `claims` holds the index this warp (or its unit) has already claimed and, with KS > 1, the one after it; on return the first
// ones it claimed that lie past this projection, which the caller passes on to the next one.
// kDep links the two projections of the MoE layer when they run in one launch: 1 = producer (done[pass] counts the
// finished items of a pass, fenced), 2 = consumer (the B fragments of an item -- the activations the producer wrote
// for that pass -- are fetched only once done[pass] has reached `need`), 0 = stand-alone.
// A consumer only ever waits for items of the first projection, and each of those is held either by a running warp (it
// was claimed before any item of the second projection) or by the warp of this grid it is statically assigned to (index <
// number of warps; the grid has at most one block per SM, so that warp becomes resident without anyone's help): the wait
// cannot deadlock; it is bounded all the same and reports through the status word.
// KS > 1: a unit of KS warps shares an item, each warp walking 1/KS of K through its own ring; at the end of an item the
// warps add their accumulators through shared memory and each stores its share of the columns.  With one warp per item a
// step takes a warp about 630 cycles at two warps per scheduler -- instruction latency, not memory: it waits 20 cycles of
// them for data -- so a gate_up item of K = 2048 is 21 us, which is also the grain of the schedule.
struct WsUnit {
  int ks, bar, n_units;              // slice, named barrier, units in the grid
  uint32_t red;                      // partial sums of the unit's first warp: [warp][mma][lane] float4
  uint32_t next_slot;                // where the unit's first warp publishes claimed items
};
struct WsClaims {
  int cur, nxt;                      // KS == 1: cur only
};
// base + rows * n bytes.  The blocks of 16 warps have 128 registers a thread and no room for the multiples of the row pitch, which
// the others keep as 64-bit values and add: there it is one multiply-add (512 experts, 2048 x 512, us with the multiples / so:
// M=32 69.4 / 68.9, M=128 121.3 / 120.3; the other shapes lose 0.3 % that way).
template <bool kMultiplyAdd>
__device__ __forceinline__ const uint8_t* ws_row(const uint8_t* base, int n, int rows) {
  if (!kMultiplyAdd) return base + (int64_t)rows * n;
  const uint8_t* p;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(p) : "r"((uint32_t)n), "r"((uint32_t)rows), "l"(base));
  return p;
}
template <bool kSilu, int kDep, int kS = kWsStages, int KS = 1>
__device__ __forceinline__ void ws_phase(const GemvArgs& g, int* counter, const int base, WsClaims& claims, const WsLane& L, const WsUnit& U,
                                         int* done, const int need) {
  const int lane = L.lane, q = L.q, t = L.t;
  const int N = g.N;
  const int nblk = g.K / (32 * kS * KS);     // blocks of kS 32-wide k-steps (one turn of the ring)
  const int groups = g.n_slabs;              // 128-column groups per pass
  const int n_items = g.plan.hdr[1] * groups;
  if (claims.cur - base >= n_items) return;

  // unit w of the grid starts on item w (KS > 1: and goes on to w + units) without asking (one round trip to the counter less
  // before the first byte is requested); the counter hands out the items after those
  auto claim = [&]() {
    int v = 0;
    if (lane == 0) v = atomicAdd(counter, 1) + U.n_units;
    return __shfl_sync(0xffffffffu, v, 0);
  };
  // An item as read from its pass record: expert, group, and the pairs this lane deals with (B column q; the one or two
  // tokens whose outputs it stores).  Pairs 0..3 sit in the record, later ones in pairs[].
  struct Item {
    int e, grp, pass, pb, ps0, ps1;
    bool valid;
  };
  auto pair_of = [&](const int4& x, const int4& y, int tok) {
    if (tok >= 4) return g.plan.pairs[y.z + tok];
    return tok == 0 ? x.z : (tok == 1 ? x.w : (tok == 2 ? y.x : y.y));
  };
  auto describe = [&](int claimed) {
    Item d;
    const int it = claimed - base;
    d.valid = it < n_items;
    d.e = d.grp = d.pass = d.pb = 0;
    d.ps0 = d.ps1 = -1;
    if (!d.valid) return d;
    d.pass = it / groups;
    d.grp = it - d.pass * groups;
    const int4 x = g.plan.pass_rec[2 * d.pass], y = g.plan.pass_rec[2 * d.pass + 1];
    d.e = x.x;
    const int nt = x.y;
    // B column q = token q of the pass; columns past the last token repeat token 0 (their results are never stored)
    d.pb = pair_of(x, y, q < nt ? q : 0);
    const int s0 = kSilu ? 2 * t + (lane >> 4) : 2 * t;
    if (s0 < nt) d.ps0 = pair_of(x, y, s0);
    if (!kSilu && s0 + 1 < nt) d.ps1 = pair_of(x, y, s0 + 1);
    return d;
  };
  // consumer: the activations of an item's pass must be complete before any lane asks for them
  auto wait_pass = [&](const Item& d) {
    if (kDep == 2 && d.valid) {
      if (lane == 0) {
        volatile int* status = g.plan.hdr + 3;
        int v;
        asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(done + d.pass) : "memory");
        if (v < need && *status == 0) {
          const long long t0 = clock64();
          do {
            asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(done + d.pass) : "memory");
            if (clock64() - t0 > g.wait_cycles) {
              *status = B200FP4_MOE_STATUS_WAIT_EXPIRED;
              break;
            }
          } while (v < need);
        }
      }
      __syncwarp();
    }
  };
  // this lane's copy sources at k-step 0 of an item
  struct Fetch {
    const uint8_t *pc, *pm, *ps;
    const __half* pb;
    bool valid;
  };
  auto sources = [&](const Item& d) {
    Fetch f;
    f.valid = d.valid;
    f.pc = f.pm = f.ps = nullptr;
    f.pb = nullptr;
    if (!d.valid) return f;
    const uint32_t pr = (uint32_t)d.pb;
    const int64_t row = g.a_magic ? (int64_t)__umulhi(pr, g.a_magic) : (int64_t)pr;
    f.pb = g.A + row * g.lda + t * 8;
    int col;
    if (kSilu) col = L.fc < 4 ? d.grp * 64 + L.fc * 16 : g.inter + d.grp * 64 + (L.fc - 4) * 16;
    else col = d.grp * 128 + L.fc * 16;
    const int64_t lane_off = (int64_t)L.fr * N + col;
    const int step0 = KS > 1 ? U.ks * (nblk * kS) : 0;       // first k-step of this warp's slice
    f.pb += step0 * 32;
    f.pc = g.w.comp + ((int64_t)d.e * g.w.comp_e + (int64_t)step0 * 8 * N + lane_off);
    f.pm = g.w.meta + ((int64_t)d.e * g.w.meta_e + (int64_t)step0 * 4 * N + lane_off);
    f.ps = g.w.scale + ((int64_t)d.e * g.w.scale_e + (int64_t)step0 * 2 * N + lane_off);
    return f;
  };
  auto row_at = [&](const uint8_t* base, int rows) { return ws_row<kS == kWsStages && KS == 1>(base, N, rows); };
  // copies of k-step `u` (relative to f) into ring slot u; always one commit group, so that the wait counts stay fixed
  auto fetch_weights = [&](const Fetch& f, int u) {
    if (f.valid) {
      const uint32_t dst = L.ring + (uint32_t)u * kWsStageBytes;
      cp_async16_s(dst + L.d_comp, row_at(f.pc, u * 8));
      cp_async16_s(dst + 512u + L.d_comp, row_at(f.pc, u * 8 + 4));
      cp_async16_s(dst + L.d_meta, row_at(f.pm, u * 4));
      if (lane < 16) cp_async16_s(dst + L.d_scale, row_at(f.ps, u * 2));
    }
  };
  auto fetch_b = [&](const Fetch& f, int u) {
    if (f.valid) cp_async16_s(L.ring + (uint32_t)u * kWsStageBytes + L.d_b, f.pb + u * 32);
    cp_async_commit();
  };
  auto fetch = [&](const Fetch& f, int u) {
    fetch_weights(f, u);
    fetch_b(f, u);
  };
  auto advance = [&](Fetch& f) {     // kS k-steps on
    f.pc = row_at(f.pc, 8 * kS);
    f.pm = row_at(f.pm, 4 * kS);
    f.ps = row_at(f.ps, 2 * kS);
    f.pb += 32 * kS;
  };

  // The first kS k-steps of the first item.  Weights are requested before the activations they meet are known to be there.
  Item cur = describe(claims.cur);
  Fetch F = sources(cur);
#pragma unroll
  for (int u = 0; u < kS; ++u) fetch_weights(F, u);
  wait_pass(cur);
#pragma unroll
  for (int u = 0; u < kS; ++u) fetch_b(F, u);
  advance(F);

  while (true) {
    int pending = 0;                           // the item after the next, on its way to the unit's first warp
    if constexpr (KS == 1) claims.nxt = claim();
    else if (U.ks == 0 && lane == 0) pending = atomicAdd(counter, 1) + 2 * U.n_units;
    const Item nxt = describe(claims.nxt);
    const float gmul = g.w.g[cur.e];
    float acc[8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[j][k] = 0.f;

    for (int b = 0; b < nblk; ++b) {
      if (b == nblk - 1) {                     // the last block of an item prefetches the first block of the next one
        wait_pass(nxt);
        F = sources(nxt);
      }
#pragma unroll
      for (int u = 0; u < kS; ++u) {
        cp_async_wait<kS - 1>();
        __syncwarp();
        const WsStep w = ws_load_step(L, L.ring + (uint32_t)u * kWsStageBytes);
        __syncwarp();                // lane 0 may come from a branch of its own: no lane refills the slot before all have read it
        fetch(F, u);                 // k-step kS ahead, into the slot that was just read
        ws_mma_step(acc, w);
      }
      advance(F);
    }

    int after_next = 0;
    if constexpr (KS > 1) {
      // add the K-slices; this warp ends up with the mmas [ks * 8 / KS, +8 / KS), that is column pairs m and m + 4 of every
      // quad's eight for m in [ks * 4 / KS, +4 / KS)
      constexpr int kM = 4 / KS;
      auto unit_barrier = [&]() {
        __syncwarp();                          // bar.sync takes whole warps
        asm volatile("bar.sync %0, %1;" ::"r"(U.bar), "n"(32 * KS) : "memory");
      };
      const uint32_t mine = U.red + (uint32_t)U.ks * 4096u + (uint32_t)lane * 16u;
      unit_barrier();                          // the sums of the item before have been read
      if (U.ks == 0 && lane == 0) asm volatile("st.shared.u32 [%0], %1;" ::"r"(U.next_slot), "r"(pending) : "memory");
#pragma unroll
      for (int j = 0; j < 8; ++j) sts128f_at(mine + (uint32_t)j * 512u, acc[j][0], acc[j][1], acc[j][2], acc[j][3]);
      unit_barrier();
      after_next = (int)lds32_at(U.next_slot);
      float v[2 * kM][4];
#pragma unroll
      for (int jj = 0; jj < 2 * kM; ++jj) {
        const uint32_t at = U.red + (uint32_t)(U.ks * 2 * kM + jj) * 512u + (uint32_t)lane * 16u;
        float4 sum = lds128f_at(at);
#pragma unroll
        for (int s = 1; s < KS; ++s) {
          const float4 x = lds128f_at(at + (uint32_t)s * 4096u);
          sum.x += x.x;
          sum.y += x.y;
          sum.z += x.z;
          sum.w += x.w;
        }
        v[jj][0] = sum.x * gmul; v[jj][1] = sum.y * gmul; v[jj][2] = sum.z * gmul; v[jj][3] = sum.w * gmul;
      }
      const int m0 = U.ks * kM;
      if (kSilu) {
        const int hi = lane >> 4;              // as below: the half-warps swap one token's values
        uint32_t words[2 * kM];
#pragma unroll
        for (int jj = 0; jj < 2 * kM; ++jj) {
          float a[2];
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const float keep = hi ? v[jj][2 * r + 1] : v[jj][2 * r], send = hi ? v[jj][2 * r] : v[jj][2 * r + 1];
            const float recv = __shfl_xor_sync(0xffffffffu, send, 16);
            const float gate = hi ? recv : keep, up = hi ? keep : recv;
            a[r] = gate / (1.0f + __expf(-gate)) * up;
          }
          const __half2 hv = __floats2half2_rn(a[0], a[1]);
          words[jj] = *reinterpret_cast<const uint32_t*>(&hv);
        }
        if (cur.ps0 >= 0) {
          __half* dst = reinterpret_cast<__half*>(g.out) + (int64_t)cur.ps0 * g.ldo + (cur.grp * 2 + ((q & 3) >> 1)) * 32 + 4 * (q & 1) + 8 * m0;
#pragma unroll
          for (int i = 0; i < kM; ++i) *reinterpret_cast<uint2*>(dst + 8 * i) = make_uint2(words[2 * i], words[2 * i + 1]);
        }
      } else {
#pragma unroll
        for (int b2 = 0; b2 < 2; ++b2) {
          const int pair = b2 ? cur.ps1 : cur.ps0;
          if (pair < 0) continue;
          float* dst = reinterpret_cast<float*>(g.out) + (int64_t)pair * g.ldo + cur.grp * 128 + q * 16 + 2 * m0;     // fp32 results only
          if constexpr (KS == 2) {
            *reinterpret_cast<float4*>(dst) = make_float4(v[0][b2], v[0][2 + b2], v[2][b2], v[2][2 + b2]);
            *reinterpret_cast<float4*>(dst + 8) = make_float4(v[1][b2], v[1][2 + b2], v[3][b2], v[3][2 + b2]);
          } else {
            *reinterpret_cast<float2*>(dst) = make_float2(v[0][b2], v[0][2 + b2]);
            *reinterpret_cast<float2*>(dst + 8) = make_float2(v[1][b2], v[1][2 + b2]);
          }
        }
      }
    } else {
    // ---- epilogue from registers.  Column 2h + r of the quad's 16 columns for token 2t + b is acc[kJ[h]][2r + b].
    constexpr int kJ[8] = {0, 2, 4, 6, 1, 3, 5, 7};
    if (kSilu) {
      const int hi = lane >> 4;                       // lanes 0..15 hold gate columns, lanes 16..31 the matching up columns
      uint32_t words[8];
#pragma unroll
      for (int h = 0; h < 8; ++h) {
        float a[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          // each half of the warp finishes one of the quad's two tokens: it keeps its own value for that token and
          // sends the other token's value to the lane that holds the matching gate / up column
          const float keep = hi ? acc[kJ[h]][2 * r + 1] : acc[kJ[h]][2 * r];
          const float send = hi ? acc[kJ[h]][2 * r] : acc[kJ[h]][2 * r + 1];
          const float recv = __shfl_xor_sync(0xffffffffu, send, 16);
          const float gate = (hi ? recv : keep) * gmul, up = (hi ? keep : recv) * gmul;
          a[r] = gate / (1.0f + __expf(-gate)) * up;
        }
        const __half2 hv = __floats2half2_rn(a[0], a[1]);
        words[h] = *reinterpret_cast<const uint32_t*>(&hv);
      }
      if (cur.ps0 >= 0) {
        // fragment order: this lane's 16 gate columns are words 8(q%2) + m, m = 0..7, of the 32-column group
        // 2 grp + (q%4)/2; word w goes to position 4(w%4) + w/4, so words m and m+4 are neighbours
        __half* dst = reinterpret_cast<__half*>(g.out) + (int64_t)cur.ps0 * g.ldo + (cur.grp * 2 + ((q & 3) >> 1)) * 32 + 4 * (q & 1);
#pragma unroll
        for (int m = 0; m < 4; ++m) *reinterpret_cast<uint2*>(dst + 8 * m) = make_uint2(words[m], words[m + 4]);
      }
    } else {
#pragma unroll
      for (int b2 = 0; b2 < 2; ++b2) {
        const int pair = b2 ? cur.ps1 : cur.ps0;
        if (pair >= 0) {
          const int64_t o = (int64_t)pair * g.ldo + cur.grp * 128 + q * 16;
          float v[16];
#pragma unroll
          for (int h = 0; h < 8; ++h) {
            v[2 * h] = acc[kJ[h]][b2] * gmul;
            v[2 * h + 1] = acc[kJ[h]][2 + b2] * gmul;
          }
          if (g.out_dtype == B200FP4_DTYPE_F32) {
            float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(g.out) + o);
#pragma unroll
            for (int i = 0; i < 4; ++i) dst[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
          } else {
            uint32_t w[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              if (g.out_dtype == B200FP4_DTYPE_F16) {
                const __half2 hv = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
                w[i] = *reinterpret_cast<const uint32_t*>(&hv);
              } else {
                const __nv_bfloat162 bv2 = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
                w[i] = *reinterpret_cast<const uint32_t*>(&bv2);
              }
            }
            uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(g.out) + o);
            dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
            dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
          }
        }
      }
    }
    }
    if (kDep == 1) {
      // this warp's activations are stored: make them visible, then count them for the pass
      __syncwarp();
      if (lane == 0) {
        __threadfence();
        atomicAdd(done + cur.pass, 1);
      }
    }
    claims.cur = claims.nxt;
    claims.nxt = after_next;
    if (!nxt.valid) break;
    cur = nxt;
  }
  cp_async_wait<0>();
  __syncwarp();
}

// The unit of this warp and its first item(s).  Units are numbered across the blocks, so that few items sit on many SMs.
template <int kS, int kW, int KS>
__device__ __forceinline__ WsUnit ws_unit(const WsLane& L, WsClaims& claims) {
  const int warp = threadIdx.x >> 5, unit = warp / KS;
  const uint32_t ring0 = L.ring - (uint32_t)warp * (kS * kWsStageBytes), red0 = ring0 + (uint32_t)kW * (kS * kWsStageBytes);
  WsUnit u;
  u.ks = warp - unit * KS;
  u.bar = 1 + unit;
  u.n_units = (int)gridDim.x * (kW / KS);
  u.red = red0 + (uint32_t)unit * (KS * 4096u);
  u.next_slot = red0 + (uint32_t)kW * 4096u + (uint32_t)unit * 4u;
  claims.cur = unit * (int)gridDim.x + (int)blockIdx.x;
  claims.nxt = claims.cur + u.n_units;
  return u;
}
template <int kS, int kW, int KS>
constexpr size_t ws_smem_bytes() { return (size_t)kW * kS * kWsStageBytes + 128 + (KS > 1 ? (size_t)kW * 4096 + 4 * (kW / KS) : 0); }

template <bool kSilu, int kS = kWsStages, int kW = kWsWarps>
__global__ void __launch_bounds__(32 * kW, 1) sparse_gemv_ws_kernel(const GemvArgs g, int* counter) {
  extern __shared__ __align__(16) unsigned char smem[];
  pdl_wait();
  pdl_launch_dependents();
  const WsLane L = ws_lane<kS>(smem);
  WsClaims claims;
  const WsUnit U = ws_unit<kS, kW, 1>(L, claims);
  ws_phase<kSilu, 0, kS>(g, counter, 0, claims, L, U, nullptr, 0);
}

// Both projections of the MoE layer in one launch: the claim sequence runs through the gate_up items and on into the
// down items, so a warp that finds no gate_up item left starts on the down projection of passes that are complete
// instead of idling until the slowest warp of a first launch has finished and a second launch has ramped up.
// kSB: ring slots the down projection turns through (its slice of K may be shorter than a ring).
template <int kS, int kW, int KS, int kSB>
__global__ void __launch_bounds__(32 * kW, 1)
    fused_moe_ws_kernel(const GemvArgs ga, const GemvArgs gb, int* counter, int* done, int need) {
  extern __shared__ __align__(16) unsigned char smem[];
  pdl_wait();
  pdl_launch_dependents();
  const WsLane L = ws_lane<kS>(smem);
  WsClaims claims;
  const WsUnit U = ws_unit<kS, kW, KS>(L, claims);
  const int n_a = ga.plan.hdr[1] * ga.n_slabs;
  ws_phase<true, 1, kS, KS>(ga, counter, 0, claims, L, U, done, need);
  ws_phase<false, 2, kSB, KS>(gb, counter, n_a, claims, L, U, done, need);
}

// ------------------------------------------------------------------------------------------ generic

// Scalar kernel for shapes the vectorised kernel does not take (N % 16 != 0, unusual scale group
// counts) and for the dense [E, K/2, N] layout: one thread per (pair, column), fp32 throughout.
// mode 0: 2:4 compressed (SparseWeights addressing); mode 1: dense transposed codes.
__global__ void generic_gemv_kernel(SparseWeights w, int mode, const void* A, int a_bf16, int64_t lda,
                                    const int32_t* __restrict__ expert_ids, int E, void* out, int out_dtype, int P,
                                    int N, int K, int G) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  const int p = blockIdx.y;
  if (n >= N || p >= P) return;
  const int e = expert_ids[p];
  if (e < 0 || e >= E) {
    store_out(out, out_dtype, (int64_t)p * N + n, 0.f);
    return;
  }
  const float lut[8] = {0.f, 0.5f, 1.f, 1.5f, 2.f, 3.f, 4.f, 6.f};
  auto dec = [&](uint32_t nib) { float v = lut[nib & 7]; return (nib & 8) ? -v : v; };
  auto a_at = [&](int k) {
    return a_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(A)[(int64_t)p * lda + k])
                  : __half2float(reinterpret_cast<const __half*>(A)[(int64_t)p * lda + k]);
  };
  float acc = 0.f;
  if (mode == 0) {
    const int pairs_per_scale = (K / 8) / G;
    const uint8_t* comp = w.comp + (int64_t)e * w.comp_e + n;
    const uint8_t* meta = w.meta + (int64_t)e * w.meta_e + n;
    const uint8_t* scale = w.scale + (int64_t)e * w.scale_e + n;
    for (int pr = 0; pr < K / 8; ++pr) {
      const uint32_t c0 = comp[(int64_t)pr * w.comp_pair], c1 = comp[(int64_t)pr * w.comp_pair + w.comp_odd];
      const uint32_t mt = meta[(int64_t)pr * w.meta_row];
      const float s = e4m3_to_f32(scale[(int64_t)(pr / pairs_per_scale) * w.scale_row] & 0x7F);
      const int k0 = pr * 8;
      float sum = dec(c0 & 15) * a_at(k0 + (mt & 3)) + dec(c0 >> 4) * a_at(k0 + ((mt >> 2) & 3)) +
                  dec(c1 & 15) * a_at(k0 + 4 + ((mt >> 4) & 3)) + dec(c1 >> 4) * a_at(k0 + 4 + ((mt >> 6) & 3));
      acc = fmaf(sum, s, acc);
    }
  } else {
    const int k_per_scale = K / G;
    const uint8_t* dense = w.comp + (int64_t)e * w.comp_e + n;
    const uint8_t* scale = w.scale + (int64_t)e * w.scale_e + n;
    for (int r = 0; r < K / 2; ++r) {
      const uint32_t c = dense[(int64_t)r * N];
      const float s = e4m3_to_f32(scale[(int64_t)((2 * r) / k_per_scale) * w.scale_row] & 0x7F);
      acc = fmaf(dec(c & 15) * a_at(2 * r) + dec(c >> 4) * a_at(2 * r + 1), s, acc);
    }
  }
  store_out(out, out_dtype, (int64_t)p * N + n, acc * w.g[e]);
}

// Where the rows of the layer's result go when they are not one [M, H] tensor: row m is row dest_row0 + m % rows_per_dest
// of the buffer ptrs[m / rows_per_dest] (expert parallelism over peer memory: the partial rows of the tokens of rank g go
// straight into rank g's buffer).  ptrs == nullptr: the plain tensor.
struct OutScatter {
  void* const* ptrs;
  int rows_per_dest, dest_row0;
  // the layer's status word, forwarded by its last kernel (status_out may be host memory the device can address)
  int* status_out = nullptr;
  const int* status_src = nullptr;
};

// out[m, h] = sum_t weight(m,t) * down[m*topk + t, h] over pairs whose expert is local.
// One thread = four columns of one token; the rows of kRedRows slots are requested before the first is used (the kernel is
// pure latency: 2.6 MB at batch 32), the sum runs in slot order.  H % 4 == 0.  Which slots count and with what weight is read while the
// kernel before still runs: that kernel starts the next one only when all before it, the plan among them, have ended.  Lane t of every warp
// reads slot t of 32 and the warp walks over those that count: a token of an expert-parallel rank has one or two of its ten.
// Ten rows are what 64 registers hold, with which eight blocks fit an SM and 1024 of them (256 tokens, H=2048) run at once.  Every thread
// reading every slot, sixteen rows in flight (128 registers), made the layer of such a rank (64 of 512 experts) 43.8 us and 45.3 from a
// graph; so it takes 35.8 and 35.7.  The 512-expert layer eager and from a graph: one token 10.3 and 12.7 / 10.0 and 10.8, 32 tokens 68.4
// and 70.1 / 68.3 and 67.3.
constexpr int kRedThreads = 128;
constexpr int kRedRows = 10;
struct RedRouting {
  const float* topk_w;
  const int32_t* ids;
  const int32_t* expert_map;
  int64_t ld_w, ld_ids;
  int topk, global_E, E, unweighted;
};
// the slots t0 .. t0 + 31 of token m that count, and this lane's weight
__device__ __forceinline__ uint32_t slots_of(const RedRouting& r, int m, int t0, int lane, float& w) {
  const int t = t0 + lane;
  int e = -1;
  w = 1.0f;
  if (t < r.topk) {
    if (!r.unweighted) w = __ldcg(r.topk_w + (int64_t)m * r.ld_w + t);
    e = __ldcg(r.ids + (int64_t)m * r.ld_ids + t);
    if (r.expert_map != nullptr) e = (e >= 0 && e < r.global_E) ? __ldcg(r.expert_map + e) : -1;
  }
  return __ballot_sync(0xffffffffu, e >= 0 && e < r.E);
}
__global__ void __launch_bounds__(kRedThreads)
    weighted_reduce_kernel(const float* __restrict__ down, const RedRouting r, void* out, int out_dtype, int M, int H, OutScatter sc) {
  const int h = (blockIdx.x * kRedThreads + threadIdx.x) * 4, m_src = blockIdx.y, topk = r.topk, lane = threadIdx.x & 31;
  float w;
  uint32_t slots = slots_of(r, m_src, 0, lane, w);
  int slot[kRedRows];                              // the next ones of them, -1 behind the last
  auto take = [&]() {
#pragma unroll
    for (int i = 0; i < kRedRows; ++i) {
      slot[i] = slots != 0 ? __ffs(slots) - 1 : -1;
      slots &= slots - 1;
    }
  };
  take();
  pdl_wait();
  pdl_launch_dependents();
  int m = m_src;
  if (sc.status_out != nullptr && h == 0 && m == 0) *sc.status_out = *sc.status_src;
  const bool in = h < H;
  const float* rows = down + (int64_t)m_src * topk * H + h;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int t0 = 0;;) {
    float4 v[kRedRows];
#pragma unroll
    for (int i = 0; i < kRedRows; ++i)
      if (slot[i] >= 0 && in) v[i] = *reinterpret_cast<const float4*>(rows + slot[i] * H);
#pragma unroll
    for (int i = 0; i < kRedRows; ++i) {
      if (slot[i] < 0) break;
      const float wi = __shfl_sync(0xffffffffu, w, slot[i]);
      a.x += v[i].x * wi;
      a.y += v[i].y * wi;
      a.z += v[i].z * wi;
      a.w += v[i].w * wi;
    }
    while (slots == 0 && (t0 += 32) < topk) {
      slots = slots_of(r, m_src, t0, lane, w);
      rows += (int64_t)32 * H;
    }
    if (slots == 0) break;
    take();
  }
  if (!in) return;
  if (sc.ptrs != nullptr) {
    out = sc.ptrs[m / sc.rows_per_dest];
    m = sc.dest_row0 + m % sc.rows_per_dest;
  }
  store_out4(out, out_dtype, (int64_t)m * H + h, a);
}

inline dim3 reduce_grid(int64_t H, int64_t M) { return dim3((unsigned)((H + 4 * kRedThreads - 1) / (4 * kRedThreads)), (unsigned)M); }

// ------------------------------------------------------------------------------------------ host

// Optional CUDA events recorded around the two GEMV launches of the fused layer (benchmark hook).
cudaEvent_t g_prof_events[3] = {nullptr, nullptr, nullptr};

// One-launch layer: clock64 budget of a wait on a pass counter (~1 s at 2 GHz) and a diagnostic surplus added to the
// count a down-projection item waits for (b200fp4_fused_moe_set_wait_limit).
constexpr long long kDefaultWaitCycles = 2000000000LL;
long long g_wait_cycles = kDefaultWaitCycles;
int g_wait_extra_need = 0;

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

int64_t max_passes(int64_t P, int64_t E) { return (P < E ? P : E) + P / kMaxTok + 1; }

// plan layout: hdr[8] | pairs[P] | mapped[P] | (16-byte aligned) pass_rec[max_passes][2] int4
size_t plan_bytes(int64_t P, int64_t E) {
  return align_up(sizeof(int) * (size_t)(8 + 2 * P), 16) + (size_t)max_passes(P, E) * 2 * sizeof(int4);
}

Plan carve_plan(void* ws, int64_t P, int64_t E) {
  (void)E;
  int* base = reinterpret_cast<int*>(ws);
  Plan pl;
  pl.hdr = base;
  pl.pairs = base + 8;
  pl.mapped = pl.pairs + P;
  pl.pass_rec = reinterpret_cast<int4*>(reinterpret_cast<unsigned char*>(ws) + align_up(sizeof(int) * (size_t)(8 + 2 * P), 16));
  return pl;
}

struct GemvCfg {
  int nt, cols, cg, stages;
  size_t smem;
  bool ok;
};

size_t gemv_smem(int nt, int cols, int cg, int stages, bool scale8, int64_t K) {
  const int nv = scale8 ? 8 : 7;
  return (size_t)kLutBytes + (size_t)stages * nv * nt * cols + (size_t)(nt / 32) * kMaxTok * cg * cols * 4 +
         (size_t)2 * kMaxTok * K * 2;
}

// Picks slab shape and ring depth for a K.  Every thread must own >= stages-1 scale blocks per item.
// (The kernel template also builds as 512 threads x 8 columns per thread; on B200 that variant
// measured 20 % slower at batch 32 -- 177 vs 148 us per layer -- so it is not instantiated.)
GemvCfg pick_cfg(int64_t K, bool scale8) {
  GemvCfg c = {0, 0, 0, 0, 0, false};
  const int64_t KB = K / 16;
  c.nt = kThreads;
  c.cols = 16;
  c.cg = KB >= 96 ? 8 : (KB >= 16 ? 16 : 32);
  const int64_t KS = c.nt / c.cg;
  const int64_t min_blocks = KB / KS;
  if (min_blocks < 1) return c;
  for (int s = (c.cg == 32 ? 2 : 4); s >= 2; --s) {
    if (min_blocks < s - 1) continue;
    const size_t smem = gemv_smem(c.nt, c.cols, c.cg, s, scale8, K);
    if (smem <= 227 * 1024) {
      c.stages = s;
      c.smem = smem;
      c.ok = true;
      return c;
    }
  }
  return c;
}

template <int NT, int COLS, int CG, int S, bool kScale8, bool kSilu>
int launch_gemv_t(const GemvArgs& g, int64_t grid, size_t smem, cudaStream_t st) {
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    if (cudaFuncSetAttribute(sparse_gemv_kernel<NT, COLS, CG, S, kScale8, kSilu>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess) {
      cudaGetLastError();
      return B200FP4_STATUS_EXECUTION_FAILED;
    }
    attr_set[dev] = true;
  }
  sparse_gemv_kernel<NT, COLS, CG, S, kScale8, kSilu><<<(unsigned)grid, NT, smem, st>>>(g);
  return B200FP4_STATUS_SUCCESS;
}

// ---- tensor-core kernel: configuration and launch
struct MmaCfg {
  int cg, stages, tm;
  bool ok;
};

size_t mma_smem_bytes(int64_t K, int stages, int tm) {
  const size_t a_bytes = align_up((size_t)2 * tm * (2 * (size_t)K + 16), 1024);
  return 1024 + a_bytes + (size_t)(tm / 4) * kMmaRedBytes + (size_t)kMmaWarps * stages * kMmaStageBytes;
}

// `passes` is an upper bound of the number of passes (the real number is only known on the device).
// Wide items (more column groups) have less per-item work to amortise, but with few passes they leave
// SMs without an item, so small batches take the narrowest shape that is allowed.
MmaCfg pick_mma_cfg(int64_t N, int64_t K, int64_t G, int inter_silu, int64_t passes, int tm) {
  MmaCfg c = {0, 0, tm, false};
  if (G != K / 16 || K % 32 != 0) return c;
  const int order_silu[3] = {2, 4, 1}, order_plain[3] = {4, 2, 1};
  const int order_small[3] = {1, 2, 4};
  const int64_t slabs_wide = inter_silu > 0 ? inter_silu / 128 : N / 512;     // slabs per pass of the preferred wide shape
  const bool small = passes * (slabs_wide > 0 ? slabs_wide : 1) < 2 * (int64_t)sm_count();
  for (int i = 0; i < 3; ++i) {
    const int cg = small ? order_small[i] : (inter_silu > 0 ? order_silu[i] : order_plain[i]);
    const int ksl = kMmaWarps / cg;
    const bool cols_ok = inter_silu > 0 ? (inter_silu % (64 * cg) == 0 && N == 2 * (int64_t)inter_silu) : (N % (128 * cg) == 0);
    if (cols_ok && K % (32 * ksl) == 0 && K / (32 * ksl) >= 2) {
      for (int s = 5; s >= 3; s -= 2)
        if (mma_smem_bytes(K, s, tm) <= 227 * 1024 && (s - 2 < 2 * (int)(K / (32 * ksl)))) {
          c.cg = cg;
          c.stages = s;
          c.ok = true;
          return c;
        }
    }
  }
  return c;
}

template <int CG, int S, bool kSilu, int TM>
int launch_mma_t(const GemvArgs& g, int64_t grid, cudaStream_t st) {
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    if (cudaFuncSetAttribute(sparse_gemv_mma_kernel<CG, S, kSilu, TM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             227 * 1024) != cudaSuccess) {
      cudaGetLastError();
      return B200FP4_STATUS_EXECUTION_FAILED;
    }
    attr_set[dev] = true;
  }
  launch_pdl(sparse_gemv_mma_kernel<CG, S, kSilu, TM>, dim3((unsigned)grid), dim3(kMmaThreads), mma_smem_bytes(g.K, S, TM), st,
             g);
  return B200FP4_STATUS_SUCCESS;
}

template <bool kSilu>
int launch_mma(const GemvArgs& g, const MmaCfg& c, int64_t grid, cudaStream_t st) {
  if (c.tm == 8) {
    if (c.stages == 5) {
      if (c.cg == 1) return launch_mma_t<1, 5, kSilu, 8>(g, grid, st);
      if (c.cg == 2) return launch_mma_t<2, 5, kSilu, 8>(g, grid, st);
      return launch_mma_t<4, 5, kSilu, 8>(g, grid, st);
    }
    if (c.cg == 1) return launch_mma_t<1, 3, kSilu, 8>(g, grid, st);
    if (c.cg == 2) return launch_mma_t<2, 3, kSilu, 8>(g, grid, st);
    return launch_mma_t<4, 3, kSilu, 8>(g, grid, st);
  }
  if (c.stages == 5) {
    if (c.cg == 1) return launch_mma_t<1, 5, kSilu, 4>(g, grid, st);
    if (c.cg == 2) return launch_mma_t<2, 5, kSilu, 4>(g, grid, st);
    return launch_mma_t<4, 5, kSilu, 4>(g, grid, st);
  }
  if (c.cg == 1) return launch_mma_t<1, 3, kSilu, 4>(g, grid, st);
  if (c.cg == 2) return launch_mma_t<2, 3, kSilu, 4>(g, grid, st);
  return launch_mma_t<4, 3, kSilu, 4>(g, grid, st);
}

// ---- warp-scheduled tensor-core kernel: conditions and launch
// One scale per 16 k, K in whole blocks of four 32-wide steps, whole 128-column groups (SiLU: 64 gate + 64 up), and the
// reference's separate [E, rows, N] tensors (the interleaved layout goes to the general kernel).
bool ws_ok(int64_t N, int64_t K, int64_t G, int64_t inter_silu, const SparseWeights& w) {
  if (G != K / 16 || K % 128 != 0) return false;
  if (inter_silu > 0) {
    if (inter_silu % 64 != 0 || N != 2 * inter_silu) return false;
  } else if (N % 128 != 0) {
    return false;
  }
  return w.comp_pair == 2 * N && w.comp_odd == N && w.meta_row == N && w.scale_row == N;
}

// Opt a kernel in to the large dynamic shared memory, once per device; `attr_set` belongs to the caller, one array per
// kernel instantiation (instantiations share their function type, so a static in here would be shared between them).
template <typename Kernel>
bool ws_prepare(Kernel kernel, bool* attr_set, size_t smem_bytes) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return false;
  if (!attr_set[dev]) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    attr_set[dev] = true;
  }
  return true;
}

template <bool kSilu, int kS = kWsStages, int kW = kWsWarps>
int launch_ws_t(const GemvArgs& g, int* counter, int64_t max_items, cudaStream_t st) {
  static bool attr_set[64] = {false};
  constexpr size_t smem = (size_t)kW * kS * kWsStageBytes + 128;
  if (!ws_prepare(sparse_gemv_ws_kernel<kSilu, kS, kW>, attr_set, smem)) return B200FP4_STATUS_EXECUTION_FAILED;
  int64_t grid = (max_items + kW - 1) / kW;
  if (grid > (int64_t)sm_count()) grid = sm_count();
  if (grid < 1) grid = 1;
  launch_pdl(sparse_gemv_ws_kernel<kSilu, kS, kW>, dim3((unsigned)grid), dim3(32 * kW), smem, st, g, counter);
  return B200FP4_STATUS_SUCCESS;
}

GemvArgs make_args(const SparseWeights& w, const Plan& plan, const __half* A, int64_t lda, int a_div, void* out,
                   int out_dtype, int64_t ldo, int64_t N, int64_t K, int inter_silu);

// A in fragment order, plan cut into passes of eight tokens, *counter zero (the plan kernel clears it).
int run_projection_ws(const SparseWeights& w, const Plan& plan, const __half* A, int64_t lda, int a_div, void* out,
                      int out_dtype, int64_t ldo, int64_t P, int64_t N, int64_t K, int64_t E, int inter_silu,
                      int* counter, cudaStream_t st) {
  GemvArgs g = make_args(w, plan, A, lda, a_div, out, out_dtype, ldo, N, K, inter_silu);
  g.n_slabs = inter_silu > 0 ? inter_silu / 64 : (int)(N / 128);
  const int64_t items = max_passes(P, E) * g.n_slabs;
  if (K % 256 == 0)        // 8 warps x 8-stage rings (see the fused layer for the measurements)
    return inter_silu > 0 ? launch_ws_t<true, 8, 8>(g, counter, items, st) : launch_ws_t<false, 8, 8>(g, counter, items, st);
  return inter_silu > 0 ? launch_ws_t<true>(g, counter, items, st) : launch_ws_t<false>(g, counter, items, st);
}

template <int kS, int kW, int KS, int kSB = kS>
int launch_fused_ws_t(const GemvArgs& ga, const GemvArgs& gb, int* counter, int* done, int need, cudaStream_t st) {
  static bool attr_set[64] = {false};
  constexpr size_t smem = ws_smem_bytes<kS, kW, KS>();
  static_assert(smem <= 227 * 1024, "shared memory of the ring");
  if (!ws_prepare(fused_moe_ws_kernel<kS, kW, KS, kSB>, attr_set, smem)) return B200FP4_STATUS_EXECUTION_FAILED;
  launch_pdl(fused_moe_ws_kernel<kS, kW, KS, kSB>, dim3((unsigned)sm_count()), dim3(32 * kW), smem, st, ga, gb, counter, done, need);
  return B200FP4_STATUS_SUCCESS;
}

// Passes of eight tokens if the pairs fall on the experts at random (a Poisson number of pairs each): E times the sum over j of
// P(more than 8 j pairs); with many pairs the remainders are even, which makes ceil(n / 8) n / 8 + 7 / 16 on average.
double expected_passes(double pairs, double E) {
  const double mean = pairs / E;
  if (mean > 32.0) return E * (mean / 8.0 + 0.4375);
  double p = std::exp(-mean), upto = 0.0, sum = 0.0;
  for (int n = 0; n < 128 && upto < 1.0 - 1e-6; ++n) {
    upto += p;
    if (n % 8 == 0) sum += 1.0 - upto;
    p *= mean / (n + 1);
  }
  return E * sum;
}

// Block shape of the one-launch layer by the items an SM is expected to get of either projection.  Four shapes, with 3, 6, 8 or
// 16 items of an SM in work at a time; what decides is which of them has its last round of gate_up items nearly full:
//   up to 3        12 warps, four per item (1.3 where a warp's quarter of K is under 16 steps of 32: what an item costs beside
//                  its steps then counts for more than the shorter chain; H = 1024, I = 256, M = 8: 21.0 us against 18.4)
//   6 to 7.75       8 warps, one per item, rings of eight stages (the count is an expectation: at 8 a second round is as likely)
//   12 to 16       16 warps, one per item (long gate_up items, K over 2048: only beside down items of at most a sixth of their
//                  length, whose last round is short too; 128 experts, 4096, 1024, M = 48: 133 us against 127 with two per item);
//                  and from where the last rounds of both projections are short beside the rest
//   otherwise      12 warps, two per item
// Measured on B200, us per layer:
//                    experts, H, I    512, 2048, 512                          256, 2048, 1024                 128, 4096, 1024
//   M                                 1     8     16    32    64    128  256  4     16    32    64    256     8     24    64   256
//   gate_up items an SM               0.5   4.0   7.4   12.9  19.8  25.4 29.4 4.0   12.9  19.8  25.4  46.9    6.4   11.7  14.7 40.7
//   12 warps, four per item           15.9  35.5  52.2  77.6  114   143  171  34.6  77.7  105   133   236     73.9  117   152  366
//   12 warps, two per item            19.0  35.5  51.3  70.1  99.2  125  145  35.3  77.4  97.3  122   200     81.5  112   137  310
//    8 warps, one per item            24.8  34.7  48.5  69.9  100   126  146  37.7  76.2  99.9  124   204     72.8  118   139  320
//   16 warps, one per item            27.0  37.4  51.2  69.4  107   123  137  40.2  75.2  115   130   184     95.3  119   139  299
// Over 947 cases (H 1024 to 4096, I 256 to 1024, 16 to 512 experts, M 1 to 256) the shape this picks takes 0.6 % more than the best
// of the four on average and 9 % at most; lines by counts that also grew with the widths took 1.6 and 20 %.
int launch_fused_ws(const GemvArgs& ga, const GemvArgs& gb, int* counter, int* done, int64_t local_pairs, int64_t E, cudaStream_t st) {
  const int need = ga.n_slabs, more = g_wait_extra_need;       // per warp of an item: counts a pass's down items wait for
  const double passes = expected_passes((double)local_pairs, (double)E) / sm_count();
  const double up = passes * ga.n_slabs, down = passes * gb.n_slabs;
  // 32-wide steps per warp with the item shared by KS warps; whole turns of a 4-slot ring in the gate_up projection, of 4, 3 or
  // 2 slots in the down projection
  auto turns = [&](int KS) {
    const int a = ga.K / 32, b = gb.K / 32;
    if (a % (4 * KS) != 0 || b % KS != 0) return 0;
    return b / KS % 4 == 0 ? 4 : (b / KS % 3 == 0 ? 3 : (b / KS % 2 == 0 ? 2 : 0));
  };
  if (up <= (ga.K >= 4 * 16 * 32 ? 3.0 : 1.3)) {
    const int t = turns(4), n = 4 * need + more;
    if (t == 4) return launch_fused_ws_t<4, 12, 4>(ga, gb, counter, done, n, st);
    if (t == 3) return launch_fused_ws_t<4, 12, 4, 3>(ga, gb, counter, done, n, st);
    if (t == 2) return launch_fused_ws_t<4, 12, 4, 2>(ga, gb, counter, done, n, st);
  }
  if (up > 6.0 && up <= 7.75 && ga.K % 256 == 0) {
    if (gb.K % 256 == 0) return launch_fused_ws_t<8, 8, 1>(ga, gb, counter, done, need + more, st);
    return launch_fused_ws_t<8, 8, 1, 4>(ga, gb, counter, done, need + more, st);
  }
  const bool one_round = up > 12.0 && up <= 16.0 && (ga.K <= 2048 || 6 * gb.K <= ga.K);
  if (!one_round && up + down / 7.0 <= 31.0) {
    const int t = turns(2), n = 2 * need + more;
    if (t == 4) return launch_fused_ws_t<4, 12, 2>(ga, gb, counter, done, n, st);
    if (t == 3) return launch_fused_ws_t<4, 12, 2, 3>(ga, gb, counter, done, n, st);
    if (t == 2) return launch_fused_ws_t<4, 12, 2, 2>(ga, gb, counter, done, n, st);
  }
  return launch_fused_ws_t<4, 16, 1>(ga, gb, counter, done, need + more, st);
}

template <bool kScale8, bool kSilu>
int launch_gemv(const GemvArgs& g, const GemvCfg& c, int64_t grid, cudaStream_t st) {
  if (c.cg == 32) return launch_gemv_t<256, 16, 32, 2, kScale8, kSilu>(g, grid, c.smem, st);
  if (c.cg == 8) {
    if (c.stages == 4) return launch_gemv_t<256, 16, 8, 4, kScale8, kSilu>(g, grid, c.smem, st);
    if (c.stages == 3) return launch_gemv_t<256, 16, 8, 3, kScale8, kSilu>(g, grid, c.smem, st);
    return launch_gemv_t<256, 16, 8, 2, kScale8, kSilu>(g, grid, c.smem, st);
  }
  if (c.stages == 4) return launch_gemv_t<256, 16, 16, 4, kScale8, kSilu>(g, grid, c.smem, st);
  if (c.stages == 3) return launch_gemv_t<256, 16, 16, 3, kScale8, kSilu>(g, grid, c.smem, st);
  return launch_gemv_t<256, 16, 16, 2, kScale8, kSilu>(g, grid, c.smem, st);
}

bool vector_ok(int64_t N, int64_t K, int64_t G, const SparseWeights& w, const void* A, int64_t lda) {
  if (N % 16 != 0 || K % 16 != 0) return false;
  if (G != K / 16 && G != K / 8) return false;
  if (!pick_cfg(K, G == K / 8).ok) return false;
  if (!aligned(w.comp, 16) || !aligned(w.meta, 16) || !aligned(w.scale, 16) || !aligned(A, 16)) return false;
  if ((w.comp_e | w.comp_pair | w.comp_odd | w.meta_e | w.meta_row | w.scale_e | w.scale_row) % 16 != 0) return false;
  if (lda % 8 != 0) return false;
  return true;
}

int check_common(const void* A, int a_dtype, const void* out, int out_dtype, int64_t P, int64_t N, int64_t K,
                 int64_t G, int64_t E) {
  if (P < 0 || N <= 0 || K <= 0 || E <= 0 || G <= 0 || (K % 8) != 0) return B200FP4_STATUS_INVALID_VALUE;
  if ((K / 8) % G != 0) return B200FP4_STATUS_INVALID_VALUE;
  if (a_dtype != B200FP4_DTYPE_F16 && a_dtype != B200FP4_DTYPE_BF16) return B200FP4_STATUS_NOT_SUPPORTED;
  if (out_dtype != B200FP4_DTYPE_F16 && out_dtype != B200FP4_DTYPE_BF16 && out_dtype != B200FP4_DTYPE_F32)
    return B200FP4_STATUS_NOT_SUPPORTED;
  if (P > 0 && (!A || !out)) return B200FP4_STATUS_INVALID_VALUE;
  if (P > 65535 || N > (int64_t)1 << 24 || K > (int64_t)1 << 20) return B200FP4_STATUS_NOT_SUPPORTED;
  return B200FP4_STATUS_SUCCESS;
}

// Plan + (for bf16 activations) conversion to fp16 in one launch.
// conv_mode: what the extra blocks do with the activation matrix a_src (kConv*); kConvNone = nothing.
void launch_plan(const int32_t* ids, int64_t P, int64_t ids_topk, int64_t ids_ld, const int32_t* expert_map,
                 int64_t global_E, int64_t E, const Plan& plan, const void* a_src, __half* a_f16, int64_t a_rows,
                 int64_t a_cols, int64_t a_ld, cudaStream_t st, int* zero_buf = nullptr, int zero_count = 0,
                 int max_tok = kMaxTok, int conv_mode = kConvBf16) {
  int64_t chunks = 0;
  unsigned blocks = 1;
  int conv_block = kPlanThreads;      // 16-byte chunks a block copies at a time
  if (a_src == nullptr) conv_mode = kConvNone;
  if (conv_mode != kConvNone) {
    chunks = a_rows * a_cols / 8;
    // in fragment order few chunks are spread over the SMs
    if (conv_mode != kConvBf16 && chunks <= 64 * 256) conv_block = 256;
    int64_t nb = (chunks + conv_block - 1) / conv_block;
    if (nb > 2 * (int64_t)sm_count()) nb = 2 * (int64_t)sm_count();
    blocks += (unsigned)(nb < 1 ? 1 : nb);
  }
  launch_pdl(moe_plan_kernel, dim3(blocks), dim3(kPlanThreads), 0, st, ids, (int)P, expert_map, (int)global_E, (int)E, plan,
             a_src, a_f16, chunks, (int)ids_topk, ids_ld, a_cols / 8 > 0 ? a_cols / 8 : (int64_t)1, a_ld / 8, zero_buf, zero_count,
             max_tok, conv_mode, conv_block);
}

// Runs one projection for P pairs with a plan already in `plan`.  A is fp16.
GemvArgs make_args(const SparseWeights& w, const Plan& plan, const __half* A, int64_t lda, int a_div, void* out,
                   int out_dtype, int64_t ldo, int64_t N, int64_t K, int inter_silu) {
  GemvArgs g;
  g.w = w;
  g.plan = plan;
  g.A = A;
  g.lda = lda;
  g.a_div = a_div;
  g.a_magic = a_div > 1 ? (uint32_t)(((uint64_t)1 << 32) / (uint64_t)a_div) + 1u : 0u;
  g.out = out;
  g.ldo = ldo;
  g.out_dtype = out_dtype;
  g.N = (int)N;
  g.K = (int)K;
  g.inter = inter_silu;
  g.n_slabs = 1;
  g.wait_cycles = g_wait_cycles;
  return g;
}

int run_projection(const SparseWeights& w, const Plan& plan, const __half* A, int64_t lda, int a_div, void* out,
                   int out_dtype, int64_t ldo, int64_t P, int64_t N, int64_t K, int64_t G, int64_t E, int inter_silu,
                   bool meta_ordered, cudaStream_t st, int tm = kMaxTok) {
  GemvArgs g = make_args(w, plan, A, lda, a_div, out, out_dtype, ldo, N, K, inter_silu);
  const bool s8 = (G == K / 8);
  if (meta_ordered) {
    // tensor-core kernel where the shape allows it (one scale per 16 k, whole 128-column groups)
    const MmaCfg mc = pick_mma_cfg(N, K, G, inter_silu, P < E ? P : E, tm);
    if (mc.ok) {
      g.n_slabs = inter_silu > 0 ? inter_silu / (64 * mc.cg) : (int)(N / (128 * mc.cg));
      int64_t grid = max_passes(P, E) * g.n_slabs;
      if (grid > (int64_t)sm_count()) grid = sm_count();
      if (grid < 1) grid = 1;
      return inter_silu > 0 ? launch_mma<true>(g, mc, grid, st) : launch_mma<false>(g, mc, grid, st);
    }
  }
  if (tm != kMaxTok) return B200FP4_STATUS_NOT_SUPPORTED;   // the general kernel only knows four-token passes
  const GemvCfg c = pick_cfg(K, s8);
  if (!c.ok) return B200FP4_STATUS_NOT_SUPPORTED;
  const int slab = c.cg * c.cols;
  g.n_slabs = inter_silu > 0 ? (inter_silu + slab / 2 - 1) / (slab / 2) : (int)((N + slab - 1) / slab);
  int64_t grid = max_passes(P, E) * g.n_slabs;
  if (grid > (int64_t)sm_count()) grid = sm_count();
  if (grid < 1) grid = 1;
  if (inter_silu > 0) return s8 ? launch_gemv<true, true>(g, c, grid, st) : launch_gemv<false, true>(g, c, grid, st);
  return s8 ? launch_gemv<true, false>(g, c, grid, st) : launch_gemv<false, false>(g, c, grid, st);
}

int gemv_entry(const SparseWeights& w, int mode, const void* A, int a_dtype, const int32_t* expert_ids, void* out,
               int out_dtype, int64_t P, int64_t N, int64_t K, int64_t G, int64_t E, int flags, void* workspace,
               size_t ws_bytes, void* stream) {
  int rc = check_common(A, a_dtype, out, out_dtype, P, N, K, G, E);
  if (rc != B200FP4_STATUS_SUCCESS) return rc;
  if (P == 0) return B200FP4_STATUS_SUCCESS;
  if (!w.comp || !w.scale || !w.g || !expert_ids || (mode == 0 && !w.meta)) return B200FP4_STATUS_INVALID_VALUE;
  cudaStream_t st = (cudaStream_t)stream;
  const int a_bf16 = a_dtype == B200FP4_DTYPE_BF16;
  if (mode == 0 && E <= kPlanMaxExperts && vector_ok(N, K, G, w, A, K)) {
    if (!workspace || ws_bytes < b200fp4_sparse_workspace_bytes(P, K, E) || !aligned(workspace, 16))
      return B200FP4_STATUS_ALLOC_FAILED;
    Plan plan = carve_plan(workspace, P, E);
    __half* a16 = reinterpret_cast<__half*>(reinterpret_cast<unsigned char*>(workspace) + align_up(plan_bytes(P, E), 256));
    if ((flags & B200FP4_SPARSE_META_ORDERED) != 0 && ws_ok(N, K, G, 0, w)) {
      // warp-scheduled tensor-core kernel: activations copied into fragment order, eight-token passes
      launch_plan(expert_ids, P, 1, 1, nullptr, 0, E, plan, A, a16, P, K, K, st, nullptr, 0, 8,
                  a_bf16 ? kConvBf16Frag : kConvF16Frag);
      zero_unmapped_rows_kernel<<<(unsigned)P, 128, 0, st>>>(plan.mapped, (int)P, out, out_dtype, N, (int)N);
      rc = run_projection_ws(w, plan, a16, K, 1, out, out_dtype, N, P, N, K, E, 0, plan.hdr + 2, st);
      if (rc != B200FP4_STATUS_SUCCESS) return rc;
      return finish_launch(3);
    }
    launch_plan(expert_ids, P, 1, 1, nullptr, 0, E, plan, a_bf16 ? A : nullptr, a16, P, K, K, st);
    zero_unmapped_rows_kernel<<<(unsigned)P, 128, 0, st>>>(plan.mapped, (int)P, out, out_dtype, N, (int)N);
    rc = run_projection(w, plan, a_bf16 ? a16 : reinterpret_cast<const __half*>(A), K, 1, out, out_dtype, N, P, N, K,
                        G, E, 0, (flags & B200FP4_SPARSE_META_ORDERED) != 0, st);
    if (rc != B200FP4_STATUS_SUCCESS) return rc;
    return finish_launch(3);
  }
  dim3 grid((unsigned)((N + 127) / 128), (unsigned)P);
  generic_gemv_kernel<<<grid, 128, 0, st>>>(w, mode, A, a_bf16, K, expert_ids, (int)E, out, out_dtype, (int)P, (int)N,
                                            (int)K, (int)G);
  return finish_launch(1);
}

}  // namespace
}  // namespace b200fp4

using namespace b200fp4;

extern "C" size_t b200fp4_sparse_workspace_bytes(int64_t P, int64_t K, int64_t E) {
  if (P < 0 || E < 0 || K < 0) return 0;
  return align_up(plan_bytes(P, E), 256) + align_up((size_t)P * K * sizeof(__half), 256);
}

extern "C" int b200fp4_sparse_gemv(const void* A, int a_dtype, const uint8_t* B_comp_T, const uint8_t* Meta_T_pk,
                                   const uint8_t* scales_T, const float* g_scales, const int32_t* expert_ids, void* out,
                                   int out_dtype, int64_t P, int64_t N, int64_t K, int64_t G, int64_t E, int flags,
                                   void* workspace, size_t workspace_bytes, void* stream) {
  SparseWeights w;
  w.comp = B_comp_T;
  w.meta = Meta_T_pk;
  w.scale = scales_T;
  w.g = g_scales;
  w.comp_e = (K / 4) * N;
  w.comp_pair = 2 * N;
  w.comp_odd = N;
  w.meta_e = (K / 8) * N;
  w.meta_row = N;
  w.scale_e = G * N;
  w.scale_row = N;
  return gemv_entry(w, 0, A, a_dtype, expert_ids, out, out_dtype, P, N, K, G, E, flags, workspace, workspace_bytes, stream);
}

// ------------------------------------------------------------------------------------------
// Allocation-free variant of b200fp4_sparse_gemv.
//
// Some hosts must not (or cannot) hand this library a workspace: plug-ins loaded into an inference
// server whose memory pool has already claimed nearly all device memory (a late cudaMalloc fails or
// fragments the pool), and latency-critical loops that ban allocator calls because cudaMalloc and
// cudaFree synchronise the whole device.  For them the scratch of the GEMV (the pair plan and the
// fp16 copy of bf16 activations) lives in a fixed array inside the library image instead.
//
// The array exists once per GPU that loads the library and stays resident until the process exits.
// All calls on a GPU share it: it still holds the previous call's plan when the next call starts
// (harmless -- the plan kernel rewrites every word the GEMV reads, so nothing has to be cleared), and
// two calls that overlap on the GPU (different streams, or different host threads) would overwrite
// each other's plan: serialise them.
constexpr int64_t kStaticMaxPairs = 512;
constexpr int64_t kStaticMaxK = 4096;
constexpr int64_t kStaticMaxExperts = 4096;
constexpr size_t static_align(size_t v, size_t a) { return (v + a - 1) / a * a; }
constexpr size_t kStaticPlanBytes =
    static_align(sizeof(int) * (size_t)(8 + 2 * kStaticMaxPairs), 16) +
    (size_t)(kStaticMaxPairs + kStaticMaxPairs / 4 + 1) * 2 * sizeof(int4);
constexpr size_t kStaticScratchBytes =
    static_align(kStaticPlanBytes, 256) + static_align((size_t)kStaticMaxPairs * kStaticMaxK * sizeof(__half), 256);

static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

// Device address of g_static_scratch on the current device.  In host code the symbol's name is only
// a handle; the address a kernel can use comes from cudaGetSymbolAddress, asked once per device with
// that device current.
static int static_scratch_ptr(void** out) {
  static void* ptrs[64] = {nullptr};
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    cudaGetLastError();
    return B200FP4_STATUS_NOT_INITIALIZED;
  }
  if (ptrs[dev] == nullptr) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_static_scratch) != cudaSuccess || p == nullptr) {
      cudaGetLastError();
      return B200FP4_STATUS_INTERNAL_ERROR;
    }
    ptrs[dev] = p;
  }
  *out = ptrs[dev];
  return B200FP4_STATUS_SUCCESS;
}

extern "C" int b200fp4_sparse_gemv_static(const void* A, int a_dtype, const uint8_t* B_comp_T, const uint8_t* Meta_T_pk,
                                          const uint8_t* scales_T, const float* g_scales, const int32_t* expert_ids,
                                          void* out, int out_dtype, int64_t P, int64_t N, int64_t K, int64_t G, int64_t E,
                                          void* stream) {
  // sizes the fixed scratch cannot hold are refused before anything is enqueued
  if (P > kStaticMaxPairs || K > kStaticMaxK || E > kStaticMaxExperts) return B200FP4_STATUS_NOT_SUPPORTED;
  void* scratch = nullptr;
  const int rc = static_scratch_ptr(&scratch);
  if (rc != B200FP4_STATUS_SUCCESS) return rc;
  return b200fp4_sparse_gemv(A, a_dtype, B_comp_T, Meta_T_pk, scales_T, g_scales, expert_ids, out, out_dtype, P, N, K, G,
                             E, 0, scratch, kStaticScratchBytes, stream);
}

extern "C" int b200fp4_dense_gemv(const void* A, int a_dtype, const uint8_t* B_dense_T, const uint8_t* scales_T,
                                  const float* g_scales, const int32_t* expert_ids, void* out, int out_dtype, int64_t P,
                                  int64_t N, int64_t K, int64_t G, int64_t E, void* workspace, size_t workspace_bytes,
                                  void* stream) {
  if (K > 0 && G > 0 && (K % 2 != 0 || K % G != 0 || (K / G) % 2 != 0)) return B200FP4_STATUS_INVALID_VALUE;
  SparseWeights w = {};
  w.comp = B_dense_T;
  w.scale = scales_T;
  w.g = g_scales;
  w.comp_e = (K / 2) * N;
  w.scale_e = G * N;
  w.scale_row = N;
  // the dense layout has no constraint tying G to K/8; validate with a G that passes the shared check
  int rc = check_common(A, a_dtype, out, out_dtype, P, N, K, (K % 8 == 0) ? K / 8 : 1, E);
  if (rc != B200FP4_STATUS_SUCCESS) return rc;
  if (P == 0) return B200FP4_STATUS_SUCCESS;
  if (!B_dense_T || !scales_T || !g_scales || !expert_ids) return B200FP4_STATUS_INVALID_VALUE;
  (void)workspace;
  (void)workspace_bytes;
  dim3 grid((unsigned)((N + 127) / 128), (unsigned)P);
  generic_gemv_kernel<<<grid, 128, 0, (cudaStream_t)stream>>>(w, 1, A, a_dtype == B200FP4_DTYPE_BF16, K, expert_ids,
                                                              (int)E, out, out_dtype, (int)P, (int)N, (int)K, (int)G);
  return finish_launch(1);
}

extern "C" int b200fp4_sparse_packed_gemv(const void* A, int a_dtype, const uint8_t* B_packed_T, const float* g_scales,
                                          const int32_t* expert_ids, void* out, int out_dtype, int64_t P, int64_t N,
                                          int64_t K, int64_t E, void* workspace, size_t workspace_bytes, void* stream) {
  SparseWeights w;
  w.comp = B_packed_T;
  w.meta = B_packed_T ? B_packed_T + 2 * N : nullptr;
  w.scale = B_packed_T ? B_packed_T + 3 * N : nullptr;
  w.g = g_scales;
  w.comp_e = (K / 8) * 4 * N;
  w.comp_pair = 4 * N;
  w.comp_odd = N;
  w.meta_e = w.comp_e;
  w.meta_row = 4 * N;
  w.scale_e = w.comp_e;
  w.scale_row = 4 * N;
  return gemv_entry(w, 0, A, a_dtype, expert_ids, out, out_dtype, P, N, K, K / 8, E, 0, workspace, workspace_bytes, stream);
}

extern "C" void b200fp4_fused_moe_profile_events(void* before_gate_up, void* after_gate_up, void* after_down) {
  g_prof_events[0] = (cudaEvent_t)before_gate_up;
  g_prof_events[1] = (cudaEvent_t)after_gate_up;
  g_prof_events[2] = (cudaEvent_t)after_down;
}

extern "C" void b200fp4_fused_moe_set_wait_limit(int64_t cycles, int extra_need) {
  g_wait_cycles = cycles > 0 ? (long long)cycles : kDefaultWaitCycles;
  g_wait_extra_need = extra_need > 0 ? extra_need : 0;
}

extern "C" int b200fp4_fused_moe_last_status(const void* workspace, void* stream, int* status) {
  if (!workspace || !status) return B200FP4_STATUS_INVALID_VALUE;
  cudaStream_t st = (cudaStream_t)stream;
  // the status word is hdr[3] of the plan at the start of the layer's workspace
  if (cudaMemcpyAsync(status, reinterpret_cast<const int*>(workspace) + 3, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess) {
    cudaGetLastError();
    return B200FP4_STATUS_EXECUTION_FAILED;
  }
  return B200FP4_STATUS_SUCCESS;
}

extern "C" size_t b200fp4_fused_moe_workspace_bytes(int64_t M, int64_t topk, int64_t H, int64_t I, int64_t E) {
  if (M < 0 || topk <= 0 || H <= 0 || I <= 0 || E <= 0) return 0;
  const int64_t P = M * topk;
  return align_up(plan_bytes(P, E), 256) + align_up((size_t)M * H * sizeof(__half), 256) +
         align_up((size_t)P * I * sizeof(__half), 256) + align_up((size_t)P * H * sizeof(float), 256) +
         align_up((size_t)max_passes(P, E) * sizeof(int), 256);
}

// The two projections' weights as the kernels address them.
static void fused_moe_weights(const uint8_t* w13_comp, const uint8_t* w13_meta, const uint8_t* w13_scale, const float* w13_g, int64_t G13,
                              const uint8_t* w2_comp, const uint8_t* w2_meta, const uint8_t* w2_scale, const float* w2_g, int64_t G2,
                              int64_t H, int64_t I, SparseWeights& w13, SparseWeights& w2) {
  w13.comp = w13_comp; w13.meta = w13_meta; w13.scale = w13_scale; w13.g = w13_g;
  w13.comp_e = (H / 4) * 2 * I; w13.comp_pair = 4 * I; w13.comp_odd = 2 * I;
  w13.meta_e = (H / 8) * 2 * I; w13.meta_row = 2 * I; w13.scale_e = G13 * 2 * I; w13.scale_row = 2 * I;
  w2.comp = w2_comp; w2.meta = w2_meta; w2.scale = w2_scale; w2.g = w2_g;
  w2.comp_e = (I / 4) * H; w2.comp_pair = 2 * H; w2.comp_odd = H;
  w2.meta_e = (I / 8) * H; w2.meta_row = H; w2.scale_e = G2 * H; w2.scale_row = H;
}

// What the fused layer refuses, without queueing anything.
static int fused_moe_check(const void* hidden, int64_t ld_h, int h_dtype, const float* topk_weights, int64_t ld_w,
                           const int32_t* topk_ids, int64_t ld_ids, const int32_t* expert_map, int64_t global_E,
                           const SparseWeights& w13, int64_t G13, const SparseWeights& w2, int64_t G2, const void* out, int out_dtype,
                           int64_t M, int64_t topk, int64_t H, int64_t I, int64_t E, const void* workspace, size_t workspace_bytes,
                           const OutScatter& sc) {
  if (M < 0 || topk <= 0 || H <= 0 || I <= 0 || E <= 0) return B200FP4_STATUS_INVALID_VALUE;
  if (ld_h < H || ld_w < topk || ld_ids < topk || (ld_h % 8) != 0) return B200FP4_STATUS_INVALID_VALUE;
  if (sc.ptrs != nullptr && (sc.rows_per_dest <= 0 || sc.dest_row0 < 0)) return B200FP4_STATUS_INVALID_VALUE;
  if (sc.ptrs != nullptr && !out) out = workspace;      // the checks below want a non-null result pointer; it is not written
  const int64_t P = M * topk;
  int rc = check_common(hidden, h_dtype, out, out_dtype, P, 2 * I, H, G13, E);
  if (rc != B200FP4_STATUS_SUCCESS) return rc;
  rc = check_common(hidden, h_dtype, out, out_dtype, P, H, I, G2, E);
  if (rc != B200FP4_STATUS_SUCCESS) return rc;
  if (M == 0) return B200FP4_STATUS_SUCCESS;
  if (!topk_weights || !topk_ids || !w13.comp || !w13.meta || !w13.scale || !w13.g || !w2.comp || !w2.meta || !w2.scale || !w2.g)
    return B200FP4_STATUS_INVALID_VALUE;
  if (expert_map && global_E <= 0) return B200FP4_STATUS_INVALID_VALUE;
  if (E > kPlanMaxExperts) return B200FP4_STATUS_NOT_SUPPORTED;
  // the fused layer only exists in vectorised form
  if (I % 16 != 0 || !vector_ok(2 * I, H, G13, w13, hidden, ld_h) || !vector_ok(H, I, G2, w2, hidden, I))
    return B200FP4_STATUS_NOT_SUPPORTED;
  if (!workspace || !aligned(workspace, 256) || workspace_bytes < b200fp4_fused_moe_workspace_bytes(M, topk, H, I, E))
    return B200FP4_STATUS_ALLOC_FAILED;
  return B200FP4_STATUS_SUCCESS;
}

// ld_h / ld_w / ld_ids: row strides (in elements) of hidden, topk_weights and topk_ids.
static int fused_moe_impl(const void* hidden, int64_t ld_h, int h_dtype, const float* topk_weights, int64_t ld_w,
                          const int32_t* topk_ids, int64_t ld_ids, const int32_t* expert_map, int64_t global_E,
                          const uint8_t* w13_comp, const uint8_t* w13_meta, const uint8_t* w13_scale, const float* w13_g,
                          int64_t G13, const uint8_t* w2_comp, const uint8_t* w2_meta, const uint8_t* w2_scale,
                          const float* w2_g, int64_t G2, void* out, int out_dtype, int64_t M, int64_t topk, int64_t H,
                          int64_t I, int64_t E, int flags, void* workspace, size_t workspace_bytes, void* stream,
                          OutScatter sc = OutScatter{nullptr, 1, 0}) {
  SparseWeights w13, w2;
  fused_moe_weights(w13_comp, w13_meta, w13_scale, w13_g, G13, w2_comp, w2_meta, w2_scale, w2_g, G2, H, I, w13, w2);
  int rc = fused_moe_check(hidden, ld_h, h_dtype, topk_weights, ld_w, topk_ids, ld_ids, expert_map, global_E, w13, G13, w2, G2, out,
                           out_dtype, M, topk, H, I, E, workspace, workspace_bytes, sc);
  if (rc != B200FP4_STATUS_SUCCESS || M == 0) return rc;
  if (sc.ptrs != nullptr && !out) out = workspace;      // not written
  const int64_t P = M * topk;
  cudaStream_t st = (cudaStream_t)stream;
  unsigned char* ws = reinterpret_cast<unsigned char*>(workspace);
  Plan plan = carve_plan(ws, P, E);
  sc.status_src = plan.hdr + 3;
  size_t off = align_up(plan_bytes(P, E), 256);
  __half* h16 = reinterpret_cast<__half*>(ws + off);
  off += align_up((size_t)M * H * sizeof(__half), 256);
  __half* act = reinterpret_cast<__half*>(ws + off);
  off += align_up((size_t)P * I * sizeof(__half), 256);
  float* down = reinterpret_cast<float*>(ws + off);
  const bool bf = h_dtype == B200FP4_DTYPE_BF16;
  const bool ordered = (flags & B200FP4_SPARSE_META_ORDERED) != 0;
  off += align_up((size_t)P * H * sizeof(float), 256);
  int* done = reinterpret_cast<int*>(ws + off);
  const int64_t n_done = max_passes(P, E);
  // the plan leaves each pair's local expert behind: one look-up less for the sum than through expert_map
  const int unweighted = (flags & B200FP4_MOE_ROUTER_WEIGHT_ON_INPUT) ? 1 : 0;
  const RedRouting routing = {topk_weights, plan.mapped, nullptr, ld_w, topk, (int)topk, 0, (int)E, unweighted};
  const int64_t local_pairs = (expert_map && global_E > 0) ? P * E / global_E : P;      // expected

  // The warp-scheduled tensor-core kernel (passes of eight tokens, activations in fragment order from the plan kernel and
  // from the gate_up epilogue).  Both projections share one launch and one claim sequence unless
  // B200FP4_MOE_SEPARATE_LAUNCHES asks for one launch each (which takes other kernels up to 256 pairs).
  if (ordered && (P > 256 || !(flags & B200FP4_MOE_SEPARATE_LAUNCHES)) && ws_ok(2 * I, H, G13, I, w13) && ws_ok(H, I, G2, 0, w2)) {
    // few pairs, which rarely share an expert: a cluster of blocks for each
    const double local = (double)P * (expert_map && global_E > E ? (double)E / (double)global_E : 1.0);
    const int cluster = (flags & B200FP4_MOE_SEPARATE_LAUNCHES) || 2 * local_pairs > E ? 0 : moe_small_cluster(P, local, H, I);
    if (cluster > 0) {
      const MoeSmallArgs a = {w13, w2, hidden, ld_h, topk_ids, ld_ids, expert_map, (int)global_E, (int)E, (int)topk, (int)H, (int)I,
                              plan.hdr + 3, down};
      if (g_prof_events[0]) cudaEventRecord(g_prof_events[0], st);
      rc = launch_moe_small(cluster, bf, a, P, st);
      if (rc != B200FP4_STATUS_SUCCESS) return rc;
      if (g_prof_events[1]) cudaEventRecord(g_prof_events[1], st);
      if (g_prof_events[2]) cudaEventRecord(g_prof_events[2], st);
      const RedRouting by_ids = {topk_weights, topk_ids, expert_map, ld_w, ld_ids, (int)topk, (int)global_E, (int)E, unweighted};
      launch_pdl(weighted_reduce_kernel, reduce_grid(H, M), dim3(kRedThreads), 0, st, (const float*)down, by_ids, out, out_dtype, (int)M, (int)H, sc);
      return finish_launch(2);
    }
    launch_plan(topk_ids, P, topk, ld_ids, expert_map, global_E, E, plan, hidden, h16, M, H, ld_h, st, done, (int)n_done, 8,
                bf ? kConvBf16Frag : kConvF16Frag);
    if (g_prof_events[0]) cudaEventRecord(g_prof_events[0], st);
    if (!(flags & B200FP4_MOE_SEPARATE_LAUNCHES)) {
      GemvArgs ga = make_args(w13, plan, h16, H, (int)topk, act, B200FP4_DTYPE_F16, I, 2 * I, H, (int)I);
      GemvArgs gb = make_args(w2, plan, act, I, 1, down, B200FP4_DTYPE_F32, H, H, I, 0);
      ga.n_slabs = (int)(I / 64);
      gb.n_slabs = (int)(H / 128);
      rc = launch_fused_ws(ga, gb, plan.hdr + 2, done, local_pairs, E, st);
      if (rc != B200FP4_STATUS_SUCCESS) return rc;
      if (g_prof_events[1]) cudaEventRecord(g_prof_events[1], st);
    } else {
      rc = run_projection_ws(w13, plan, h16, H, (int)topk, act, B200FP4_DTYPE_F16, I, P, 2 * I, H, E, (int)I, plan.hdr + 2, st);
      if (rc != B200FP4_STATUS_SUCCESS) return rc;
      if (g_prof_events[1]) cudaEventRecord(g_prof_events[1], st);
      rc = run_projection_ws(w2, plan, act, I, 1, down, B200FP4_DTYPE_F32, H, P, H, I, E, 0, plan.hdr + 4, st);
      if (rc != B200FP4_STATUS_SUCCESS) return rc;
    }
    if (g_prof_events[2]) cudaEventRecord(g_prof_events[2], st);
    launch_pdl(weighted_reduce_kernel, reduce_grid(H, M), dim3(kRedThreads), 0, st, (const float*)down, routing, out, out_dtype, (int)M, (int)H, sc);
    return finish_launch((flags & B200FP4_MOE_SEPARATE_LAUNCHES) ? 4 : 3);
  }

  // Tokens per pass: eight when the local experts see four or more tokens each on average (large
  // batches, expert parallelism with many source ranks) and both projections have a tensor-core
  // configuration for it; four otherwise.
  const int64_t pb = P < E ? P : E;
  int tm = kMaxTok;
  if (ordered && local_pairs >= 4 * E) {
    const MmaCfg a8 = pick_mma_cfg(2 * I, H, G13, (int)I, pb, 8), b8 = pick_mma_cfg(H, I, G2, 0, pb, 8);
    if (a8.ok && b8.ok) tm = 8;
  }
  launch_plan(topk_ids, P, topk, ld_ids, expert_map, global_E, E, plan, bf ? hidden : nullptr, h16, M, H, ld_h, st, done,
              (int)n_done, tm);
  if (g_prof_events[0]) cudaEventRecord(g_prof_events[0], st);
  rc = run_projection(w13, plan, bf ? h16 : reinterpret_cast<const __half*>(hidden), bf ? H : ld_h, (int)topk, act,
                      B200FP4_DTYPE_F16, I, P, 2 * I, H, G13, E, (int)I, ordered, st, tm);
  if (rc != B200FP4_STATUS_SUCCESS) return rc;
  if (g_prof_events[1]) cudaEventRecord(g_prof_events[1], st);
  rc = run_projection(w2, plan, act, I, 1, down, B200FP4_DTYPE_F32, H, P, H, I, G2, E, 0, ordered, st, tm);
  if (rc != B200FP4_STATUS_SUCCESS) return rc;
  if (g_prof_events[2]) cudaEventRecord(g_prof_events[2], st);
  launch_pdl(weighted_reduce_kernel, reduce_grid(H, M), dim3(kRedThreads), 0, st, (const float*)down, routing, out, out_dtype, (int)M, (int)H, sc);
  return finish_launch(4);
}

extern "C" int b200fp4_fused_sparse_moe(const void* hidden, int h_dtype, const float* topk_weights,
                                        const int32_t* topk_ids, const int32_t* expert_map, int64_t global_E,
                                        const uint8_t* w13_comp, const uint8_t* w13_meta, const uint8_t* w13_scale,
                                        const float* w13_g, int64_t G13, const uint8_t* w2_comp, const uint8_t* w2_meta,
                                        const uint8_t* w2_scale, const float* w2_g, int64_t G2, void* out, int out_dtype,
                                        int64_t M, int64_t topk, int64_t H, int64_t I, int64_t E, int flags,
                                        void* workspace, size_t workspace_bytes, void* stream) {
  return fused_moe_impl(hidden, H, h_dtype, topk_weights, topk, topk_ids, topk, expert_map, global_E, w13_comp, w13_meta,
                        w13_scale, w13_g, G13, w2_comp, w2_meta, w2_scale, w2_g, G2, out, out_dtype, M, topk, H, I, E, flags,
                        workspace, workspace_bytes, stream);
}

// The layer for a caller whose activations, routing and result live in HOST memory (pinned memory makes the
// copies asynchronous): three copies in, the device entry point above, one copy out, one stream
// synchronisation.  The device workspace holds the staging buffers in front of the layer's own workspace.
static size_t host_stage_bytes(int64_t M, int64_t topk, int64_t H) {
  return 2 * align_up((size_t)M * H * sizeof(__half), 256) + 2 * align_up((size_t)M * topk * sizeof(float), 256);
}

extern "C" size_t b200fp4_fused_moe_host_workspace_bytes(int64_t M, int64_t topk, int64_t H, int64_t I, int64_t E) {
  if (M < 0 || topk <= 0 || H <= 0 || I <= 0 || E <= 0) return 0;
  return host_stage_bytes(M, topk, H) + b200fp4_fused_moe_workspace_bytes(M, topk, H, I, E);
}

namespace {
// Events that order a copy stream against the compute stream, one pair per workspace (the staging buffers they guard
// live in the workspace).  Created on first use, kept for the life of the process.
struct HostSlotEvents {
  const void* workspace;
  int device;
  cudaEvent_t loaded, consumed;
  bool used;
};
constexpr int kHostSlots = 32;
HostSlotEvents g_host_slots[kHostSlots];
int g_host_slot_count = 0;
std::mutex g_host_slot_mutex;

HostSlotEvents* host_slot_events(const void* workspace) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  std::lock_guard<std::mutex> lock(g_host_slot_mutex);
  for (int i = 0; i < g_host_slot_count; ++i)
    if (g_host_slots[i].workspace == workspace && g_host_slots[i].device == dev) return &g_host_slots[i];
  if (g_host_slot_count == kHostSlots) return nullptr;
  HostSlotEvents& e = g_host_slots[g_host_slot_count];
  if (cudaEventCreateWithFlags(&e.loaded, cudaEventDisableTiming) != cudaSuccess) return nullptr;
  if (cudaEventCreateWithFlags(&e.consumed, cudaEventDisableTiming) != cudaSuccess) {
    cudaEventDestroy(e.loaded);
    return nullptr;
  }
  e.workspace = workspace;
  e.device = dev;
  e.used = false;
  ++g_host_slot_count;
  return &e;
}
}  // namespace

// Enqueue-only form: copies in (on copy_stream when one is given, ordered against the layer by events), the layer, the
// copies out; no host synchronisation.
extern "C" int b200fp4_fused_sparse_moe_host_async(const void* hidden_host, int h_dtype, const float* topk_weights_host,
                                                   const int32_t* topk_ids_host, const int32_t* expert_map,
                                                   int64_t global_E, const uint8_t* w13_comp, const uint8_t* w13_meta,
                                                   const uint8_t* w13_scale, const float* w13_g, int64_t G13,
                                                   const uint8_t* w2_comp, const uint8_t* w2_meta, const uint8_t* w2_scale,
                                                   const float* w2_g, int64_t G2, void* out_host, int out_dtype,
                                                   int32_t* status_host, int64_t M, int64_t topk, int64_t H, int64_t I,
                                                   int64_t E, int flags, void* workspace, size_t workspace_bytes,
                                                   void* stream, void* copy_stream) {
  if (M < 0 || topk <= 0 || H <= 0 || I <= 0 || E <= 0) return B200FP4_STATUS_INVALID_VALUE;
  if (M == 0) return B200FP4_STATUS_SUCCESS;
  if (!hidden_host || !topk_weights_host || !topk_ids_host || !out_host || !workspace)
    return B200FP4_STATUS_INVALID_VALUE;
  if (out_dtype != B200FP4_DTYPE_F16 && out_dtype != B200FP4_DTYPE_BF16) return B200FP4_STATUS_NOT_SUPPORTED;
  const size_t stage = host_stage_bytes(M, topk, H);
  if (workspace_bytes < stage) return B200FP4_STATUS_INVALID_VALUE;
  const size_t nh = (size_t)M * H * sizeof(__half), nr = (size_t)M * topk * sizeof(float);
  char* d_hidden = static_cast<char*>(workspace);
  char* d_out = d_hidden + align_up(nh, 256);
  char* d_w = d_out + align_up(nh, 256);
  char* d_ids = d_w + align_up(nr, 256);
  {
    // what the layer would refuse, before the copies are queued
    SparseWeights w13, w2;
    fused_moe_weights(w13_comp, w13_meta, w13_scale, w13_g, G13, w2_comp, w2_meta, w2_scale, w2_g, G2, H, I, w13, w2);
    const int refused = fused_moe_check(d_hidden, H, h_dtype, reinterpret_cast<const float*>(d_w), topk,
                                        reinterpret_cast<const int32_t*>(d_ids), topk, expert_map, global_E, w13, G13, w2, G2, d_out,
                                        out_dtype, M, topk, H, I, E, static_cast<char*>(workspace) + stage, workspace_bytes - stage,
                                        OutScatter{nullptr, 1, 0});
    if (refused != B200FP4_STATUS_SUCCESS) return refused;
  }
  cudaStream_t st = (cudaStream_t)stream;
  cudaStream_t cs = copy_stream ? (cudaStream_t)copy_stream : st;
  HostSlotEvents* ev = nullptr;
  if (cs != st) {
    ev = host_slot_events(workspace);
    if (!ev) return B200FP4_STATUS_ALLOC_FAILED;
    // the staging buffers may still be read by the layer of the previous submission with this workspace
    if (ev->used && cudaStreamWaitEvent(cs, ev->consumed, 0) != cudaSuccess) {
      cudaGetLastError();
      return B200FP4_STATUS_EXECUTION_FAILED;
    }
  }
  if (cudaMemcpyAsync(d_ids, topk_ids_host, nr, cudaMemcpyHostToDevice, cs) != cudaSuccess ||
      cudaMemcpyAsync(d_w, topk_weights_host, nr, cudaMemcpyHostToDevice, cs) != cudaSuccess ||
      cudaMemcpyAsync(d_hidden, hidden_host, nh, cudaMemcpyHostToDevice, cs) != cudaSuccess) {
    cudaGetLastError();
    return B200FP4_STATUS_EXECUTION_FAILED;
  }
  if (ev && (cudaEventRecord(ev->loaded, cs) != cudaSuccess || cudaStreamWaitEvent(st, ev->loaded, 0) != cudaSuccess)) {
    cudaGetLastError();
    return B200FP4_STATUS_EXECUTION_FAILED;
  }
  // result rows and status word: into the staging buffer and copied out, or -- with B200FP4_MOE_HOST_DIRECT_OUT and
  // pinned memory the device can address -- stored by the layer's last kernel straight into the caller's buffers
  auto mapped_of = [](void* host) -> void* {
    cudaPointerAttributes attr;
    if (cudaPointerGetAttributes(&attr, host) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    return attr.type == cudaMemoryTypeHost ? attr.devicePointer : nullptr;
  };
  void* out_target = d_out;
  OutScatter sc{nullptr, 1, 0};
  if (flags & B200FP4_MOE_HOST_DIRECT_OUT) {
    if (void* mapped = mapped_of(out_host)) out_target = mapped;
    if (status_host) sc.status_out = static_cast<int*>(mapped_of(status_host));
  }
  const int rc = fused_moe_impl(d_hidden, H, h_dtype, reinterpret_cast<const float*>(d_w), topk,
                                reinterpret_cast<const int32_t*>(d_ids), topk, expert_map, global_E, w13_comp, w13_meta,
                                w13_scale, w13_g, G13, w2_comp, w2_meta, w2_scale, w2_g, G2, out_target, out_dtype, M, topk, H,
                                I, E, flags & ~B200FP4_MOE_HOST_DIRECT_OUT, static_cast<char*>(workspace) + stage,
                                workspace_bytes - stage, stream, sc);
  if (rc != B200FP4_STATUS_SUCCESS) return rc;
  if (ev) {
    if (cudaEventRecord(ev->consumed, st) != cudaSuccess) {
      cudaGetLastError();
      return B200FP4_STATUS_EXECUTION_FAILED;
    }
    ev->used = true;
  }
  // the layer's status word (hdr[3] of its plan) comes back with the result
  if ((out_target == d_out && cudaMemcpyAsync(out_host, d_out, nh, cudaMemcpyDeviceToHost, st) != cudaSuccess) ||
      (status_host && !sc.status_out && cudaMemcpyAsync(status_host, reinterpret_cast<const int*>(static_cast<char*>(workspace) + stage) + 3,
                                      sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess)) {
    cudaGetLastError();
    return B200FP4_STATUS_EXECUTION_FAILED;
  }
  return B200FP4_STATUS_SUCCESS;
}

extern "C" int b200fp4_fused_sparse_moe_host(const void* hidden_host, int h_dtype, const float* topk_weights_host,
                                             const int32_t* topk_ids_host, const int32_t* expert_map, int64_t global_E,
                                             const uint8_t* w13_comp, const uint8_t* w13_meta, const uint8_t* w13_scale,
                                             const float* w13_g, int64_t G13, const uint8_t* w2_comp,
                                             const uint8_t* w2_meta, const uint8_t* w2_scale, const float* w2_g,
                                             int64_t G2, void* out_host, int out_dtype, int64_t M, int64_t topk,
                                             int64_t H, int64_t I, int64_t E, int flags, void* workspace,
                                             size_t workspace_bytes, void* stream) {
  if (M == 0 && topk > 0 && H > 0 && I > 0 && E > 0) return B200FP4_STATUS_SUCCESS;
  int moe_status = 0;
  const int rc = b200fp4_fused_sparse_moe_host_async(hidden_host, h_dtype, topk_weights_host, topk_ids_host, expert_map,
                                                     global_E, w13_comp, w13_meta, w13_scale, w13_g, G13, w2_comp, w2_meta,
                                                     w2_scale, w2_g, G2, out_host, out_dtype, &moe_status, M, topk, H, I, E,
                                                     flags, workspace, workspace_bytes, stream, nullptr);
  if (rc != B200FP4_STATUS_SUCCESS) return rc;
  if (cudaStreamSynchronize((cudaStream_t)stream) != cudaSuccess) {
    cudaGetLastError();
    return B200FP4_STATUS_EXECUTION_FAILED;
  }
  return moe_status == 0 ? B200FP4_STATUS_SUCCESS : B200FP4_STATUS_INTERNAL_ERROR;
}

// ------------------------------------------------------------------------------------------ expert parallel

// One record per token: [H activations (16-bit) | topk expert ids (i32) | topk router weights (f32)].
extern "C" size_t b200fp4_ep_record_bytes(int64_t H, int64_t topk) {
  if (H <= 0 || topk <= 0) return 0;
  return align_up((size_t)H * 2 + (size_t)topk * 8, 16);
}

namespace b200fp4 {
namespace {
// out[g][b] = record of token b, for every destination rank g (fixed-capacity dispatch slots)
__global__ void ep_pack_kernel(const uint4* __restrict__ hidden, const int32_t* __restrict__ ids,
                               const float* __restrict__ w, int B, int H, int topk, int G, int64_t rec_chunks,
                               uint4* __restrict__ out) {
  const int b = blockIdx.x;
  const int h_chunks = H / 8;
  __shared__ uint4 s_tail[64];
  const int tail_chunks = (int)rec_chunks - h_chunks;
  if (threadIdx.x < tail_chunks * 4) {
    const int i = threadIdx.x;            // 32-bit word index inside the tail: ids first, then weights
    uint32_t v = 0;
    if (i < topk) v = (uint32_t)ids[(int64_t)b * topk + i];
    else if (i < 2 * topk) v = __float_as_uint(w[(int64_t)b * topk + i - topk]);
    reinterpret_cast<uint32_t*>(s_tail)[i] = v;
  }
  __syncthreads();
  for (int c = threadIdx.x; c < rec_chunks; c += blockDim.x) {
    const uint4 v = c < h_chunks ? hidden[(int64_t)b * h_chunks + c] : s_tail[c - h_chunks];
    for (int g = 0; g < G; ++g) out[((int64_t)g * B + b) * rec_chunks + c] = v;
  }
}

// out[b, :] = sum over ranks g of parts[g][b, :] accumulated in fp32
template <typename T>
__global__ void ep_combine_kernel(const T* __restrict__ parts, int B, int H, int G, T* __restrict__ out) {
  const int64_t n = (int64_t)B * H;
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 2; i < n; i += (int64_t)gridDim.x * blockDim.x * 2) {
    float a0 = 0.f, a1 = 0.f;
    for (int g = 0; g < G; ++g) {
      a0 += to_f32<T>(parts[(int64_t)g * n + i]);
      a1 += to_f32<T>(parts[(int64_t)g * n + i + 1]);
    }
    out[i] = from_f32<T>(a0);
    out[i + 1] = from_f32<T>(a1);
  }
}
}  // namespace
}  // namespace b200fp4

extern "C" int b200fp4_ep_pack(const void* hidden, const int32_t* topk_ids, const float* topk_weights, int64_t B,
                               int64_t H, int64_t topk, int64_t G, void* records, void* stream) {
  if (B < 0 || H <= 0 || (H % 8) != 0 || topk <= 0 || topk > 64 || G <= 0) return B200FP4_STATUS_INVALID_VALUE;
  if (B == 0) return B200FP4_STATUS_SUCCESS;
  if (!hidden || !topk_ids || !topk_weights || !records || !aligned(hidden, 16) || !aligned(records, 16))
    return B200FP4_STATUS_INVALID_VALUE;
  const int64_t rec_chunks = (int64_t)b200fp4_ep_record_bytes(H, topk) / 16;
  ep_pack_kernel<<<(unsigned)B, 256, 0, (cudaStream_t)stream>>>(reinterpret_cast<const uint4*>(hidden), topk_ids,
                                                               topk_weights, (int)B, (int)H, (int)topk, (int)G,
                                                               rec_chunks, reinterpret_cast<uint4*>(records));
  return finish_launch(1);
}

extern "C" int b200fp4_ep_combine(const void* parts, int dtype, int64_t B, int64_t H, int64_t G, void* out, void* stream) {
  if (B < 0 || H <= 0 || (H % 2) != 0 || G <= 0) return B200FP4_STATUS_INVALID_VALUE;
  if (dtype != B200FP4_DTYPE_BF16 && dtype != B200FP4_DTYPE_F16) return B200FP4_STATUS_NOT_SUPPORTED;
  if (B == 0) return B200FP4_STATUS_SUCCESS;
  if (!parts || !out) return B200FP4_STATUS_INVALID_VALUE;
  int64_t blocks = (B * H / 2 + 255) / 256;
  if (blocks > 4 * (int64_t)sm_count()) blocks = 4 * (int64_t)sm_count();
  if (dtype == B200FP4_DTYPE_BF16)
    ep_combine_kernel<__nv_bfloat16><<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(
        reinterpret_cast<const __nv_bfloat16*>(parts), (int)B, (int)H, (int)G, reinterpret_cast<__nv_bfloat16*>(out));
  else
    ep_combine_kernel<__half><<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(
        reinterpret_cast<const __half*>(parts), (int)B, (int)H, (int)G, reinterpret_cast<__half*>(out));
  return finish_launch(1);
}

// The fused layer over received dispatch records ([T] records of record_bytes each, as written by
// b200fp4_ep_pack on the source ranks): activations, ids and weights are read in place.
extern "C" int b200fp4_fused_sparse_moe_records(const void* records, int64_t record_bytes, int h_dtype,
                                                const int32_t* expert_map, int64_t global_E, const uint8_t* w13_comp,
                                                const uint8_t* w13_meta, const uint8_t* w13_scale, const float* w13_g,
                                                int64_t G13, const uint8_t* w2_comp, const uint8_t* w2_meta,
                                                const uint8_t* w2_scale, const float* w2_g, int64_t G2, void* out,
                                                int out_dtype, int64_t T, int64_t topk, int64_t H, int64_t I, int64_t E,
                                                int flags, void* workspace, size_t workspace_bytes, void* stream) {
  if (!records || record_bytes != (int64_t)b200fp4_ep_record_bytes(H, topk)) return B200FP4_STATUS_INVALID_VALUE;
  const unsigned char* r = reinterpret_cast<const unsigned char*>(records);
  return fused_moe_impl(r, record_bytes / 2, h_dtype, reinterpret_cast<const float*>(r + H * 2 + topk * 4),
                        record_bytes / 4, reinterpret_cast<const int32_t*>(r + H * 2), record_bytes / 4, expert_map,
                        global_E, w13_comp, w13_meta, w13_scale, w13_g, G13, w2_comp, w2_meta, w2_scale, w2_g, G2, out,
                        out_dtype, T, topk, H, I, E, flags & ~B200FP4_MOE_ROUTER_WEIGHT_ON_INPUT, workspace, workspace_bytes,
                        stream);
}

// The same with the result scattered over several buffers: row m (token m of the T received records) goes to row
// dest_row0 + m % rows_per_dest of the buffer out_ptrs[m / rows_per_dest].  out_ptrs is a DEVICE array of T /
// rows_per_dest pointers, which may point into peer GPUs' memory (plain stores over NVLink).
extern "C" int b200fp4_fused_sparse_moe_records_scatter(
    const void* records, int64_t record_bytes, int h_dtype, const int32_t* expert_map, int64_t global_E,
    const uint8_t* w13_comp, const uint8_t* w13_meta, const uint8_t* w13_scale, const float* w13_g, int64_t G13,
    const uint8_t* w2_comp, const uint8_t* w2_meta, const uint8_t* w2_scale, const float* w2_g, int64_t G2,
    void* const* out_ptrs, int64_t rows_per_dest, int64_t dest_row0, int out_dtype, int64_t T, int64_t topk, int64_t H, int64_t I,
    int64_t E, int flags, void* workspace, size_t workspace_bytes, void* stream) {
  if (!records || record_bytes != (int64_t)b200fp4_ep_record_bytes(H, topk) || !out_ptrs) return B200FP4_STATUS_INVALID_VALUE;
  if (rows_per_dest <= 0 || rows_per_dest > 0x7FFFFFFF || dest_row0 < 0 || dest_row0 > 0x7FFFFFFF) return B200FP4_STATUS_INVALID_VALUE;
  const unsigned char* r = reinterpret_cast<const unsigned char*>(records);
  OutScatter sc{out_ptrs, (int)rows_per_dest, (int)dest_row0};
  return fused_moe_impl(r, record_bytes / 2, h_dtype, reinterpret_cast<const float*>(r + H * 2 + topk * 4), record_bytes / 4,
                        reinterpret_cast<const int32_t*>(r + H * 2), record_bytes / 4, expert_map, global_E, w13_comp, w13_meta,
                        w13_scale, w13_g, G13, w2_comp, w2_meta, w2_scale, w2_g, G2, nullptr, out_dtype, T, topk, H, I, E,
                        flags & ~B200FP4_MOE_ROUTER_WEIGHT_ON_INPUT, workspace, workspace_bytes, stream, sc);
}
