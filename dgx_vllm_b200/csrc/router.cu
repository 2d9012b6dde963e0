// MoE router for decode: gate projection (16-bit weights), softmax over the experts, top-k, renormalisation.
//
// The reference leaves routing to vLLM (its benches build it in torch: softmax of the gate logits, topk, weights
// divided by their sum -- sparse_fp4_kernel/bench_moe_layer_e2e.py:230-236); here it is one or two small kernels whose
// outputs (topk_weights f32, topk_ids i32) are exactly the device tensors the fused MoE layer and the expert-parallel
// dispatch take, so no host round trip sits between the router and the experts.
//   router_cluster_kernel  up to 64 tokens: projection (mma.sync, operands straight from global memory into fragments), exchange of
//                          the logits through distributed shared memory and selection in one launch
//   router_slices_kernel   up to 32 tokens and a gate of many bytes: the same products with K split over blocks of 16 experts each
//   router_gemm_kernel     larger batches: 128 tokens x 128 or 256 experts per CTA on tcgen05 (kind::f16, fp32 accumulators
//                          in tensor memory), operands by TMA; bound by L2 -> shared-memory bandwidth
//   router_topk_kernel     one warp per token: adds the K-slices of its logits in a fixed order, then k rounds of warp-wide
//                          arg-max (ties -> lower expert id), weights exp(l - max) normalised over the selected experts
//                          (or over all of them)
#include "sm100_ptx.cuh"

namespace b200fp4 {
namespace {

// ------------------------------------------------------------------------------------------ small batches, one kernel

constexpr int kRcWarps = 16;
constexpr int kRcThreads = 32 * kRcWarps;
constexpr int kRtPerLane = 32;         // experts per lane of a warp that selects: 1024

template <typename T>
__device__ __forceinline__ void mma_m16n8k16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                             uint32_t b1);
template <>
__device__ __forceinline__ void mma_m16n8k16<__nv_bfloat16>(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                            uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void mma_m16n8k16<__half>(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                     uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// ------------------------------------------------------------------------------------------ few tokens, large gates

constexpr int kRsWarps = 8;
constexpr int kRsThreads = 32 * kRsWarps;

// parts[z][m][e] = sum over the k of slice z of hidden[m][k] * gate_w[e][k].
// Block = experts [16 x, +16) x tokens [8 NT y, +8 NT), slice z of K; its warps take 64-wide pieces of K in turn.  In a 32-wide
// step lane (g, t) = (lane / 4, lane % 4) loads the 8 elements at k = 8t of rows g and g + 8 (experts) and g (tokens): the
// order of k inside a product sum is free, so elements 0-3 of the 8 serve as the lane's k of one mma and 4-7 as those of
// another, on both sides alike.  Every SM reads its share of the gate once, whatever the number of experts; a second launch selects.
template <typename T, int NT>
__global__ void __launch_bounds__(kRsThreads)
    router_slices_kernel(const T* __restrict__ hidden, int64_t ld_h, const T* __restrict__ gate_w, int M, int H, int E,
                         int* __restrict__ status, float* __restrict__ parts) {
  __shared__ float s_part[kRsWarps][16][8 * NT + 1];
  pdl_wait();
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int e0 = blockIdx.x * 16, m0 = blockIdx.y * 8 * NT;
  if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && threadIdx.x == 0) *status = 0;
  float acc[NT][4];
#pragma unroll
  for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
  const T* wa = gate_w + (int64_t)min(e0 + g, E - 1) * H;            // rows past the end repeat the last: never stored
  const T* wb = gate_w + (int64_t)min(e0 + g + 8, E - 1) * H;
  const T* x[NT];
#pragma unroll
  for (int n = 0; n < NT; ++n) x[n] = hidden + (int64_t)min(m0 + 8 * n + g, M - 1) * ld_h;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  for (int k0 = 64 * (blockIdx.z * kRsWarps + warp); k0 < H; k0 += 64 * kRsWarps * gridDim.z) {
    uint4 a[2][2], b[2][NT];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int k = k0 + 32 * s + 8 * t;
      const bool in = k < H;
      a[s][0] = in ? ldg_stream_u4(wa + k) : zero;
      a[s][1] = in ? ldg_stream_u4(wb + k) : zero;
#pragma unroll
      for (int n = 0; n < NT; ++n) b[s][n] = in ? *reinterpret_cast<const uint4*>(x[n] + k) : zero;
    }
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        mma_m16n8k16<T>(acc[n], a[s][0].x, a[s][1].x, a[s][0].y, a[s][1].y, b[s][n].x, b[s][n].y);
        mma_m16n8k16<T>(acc[n], a[s][0].z, a[s][1].z, a[s][0].w, a[s][1].w, b[s][n].z, b[s][n].w);
      }
  }
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    s_part[warp][g][8 * n + 2 * t] = acc[n][0];
    s_part[warp][g][8 * n + 2 * t + 1] = acc[n][1];
    s_part[warp][g + 8][8 * n + 2 * t] = acc[n][2];
    s_part[warp][g + 8][8 * n + 2 * t + 1] = acc[n][3];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 16 * 8 * NT; i += kRsThreads) {
    const int r = i & 15, c = i >> 4;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < kRsWarps; ++w) v += s_part[w][r][c];
    if (e0 + r < E && m0 + c < M) parts[((int64_t)blockIdx.z * M + m0 + c) * E + e0 + r] = v;
  }
}

// ------------------------------------------------------------------------------------------ projection, larger batches

constexpr int kRgThreads = 192;              // warp 0 TMA, warp 1 MMA and tensor memory, warps 2-5 epilogue
constexpr int kRgStages = 4;
constexpr int kRgK = 64;                     // elements per stage: 128-byte rows

template <int BN>
struct RouterGemm {
  static constexpr int kStageA = 128 * 128, kStageB = BN * 128, kStage = kStageA + kStageB;
  static constexpr size_t kSmem = (size_t)kRgStages * kStage + 1024 + 256;
};

__device__ __forceinline__ void tcgen05_mma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// parts[z][m][e] = the sum over the k of K-slice z of hidden[m][k] * gate_w[e][k], for the tile of 128 tokens (blockIdx.y)
// x BN experts (blockIdx.x).  Rows and columns past the tensors are filled with zeros by the copies and not stored.
template <int BN>
__global__ void __launch_bounds__(kRgThreads, 1)
    router_gemm_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, int M, int H, int E,
                       uint32_t idesc, int* __restrict__ status, float* __restrict__ parts) {
  using C = RouterGemm<BN>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kRgStages * C::kStage);
  uint64_t* empty_bar = full_bar + kRgStages;
  uint64_t* acc_full = empty_bar + kRgStages;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(acc_full + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.y * 128, e0 = blockIdx.x * BN;
  const int steps = (H + kRgK - 1) / kRgK;
  const int first = (int)((int64_t)steps * blockIdx.z / gridDim.z), n_steps = (int)((int64_t)steps * (blockIdx.z + 1) / gridDim.z) - first;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kRgStages; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    mbar_init(smem_u32(acc_full), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_ptr_smem)), "r"((uint32_t)BN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = *tmem_ptr_smem;
  pdl_wait();
  pdl_launch_dependents();
  if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && threadIdx.x == 0) *status = 0;    // a wait writes it only after ~1 s
  if (warp == 0) {
    const bool elected = elect_one();
    for (int i = 0; i < n_steps; ++i) {
      const uint32_t s = i % kRgStages, ph = (i / kRgStages) & 1;
      if (!mbar_wait_warp(smem_u32(&empty_bar[s]), ph ^ 1, status, 31)) break;
      if (elected) {
        unsigned char* st = smem + s * C::kStage;
        const uint32_t bar = smem_u32(&full_bar[s]);
        mbar_expect_tx(bar, C::kStage);
        tma_load_2d(smem_u32(st), &map_x, (first + i) * 128, m0, bar);
        tma_load_2d(smem_u32(st + C::kStageA), &map_w, (first + i) * 128, e0, bar);
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    const bool elected = elect_one();
    for (int i = 0; i < n_steps; ++i) {
      const uint32_t s = i % kRgStages, ph = (i / kRgStages) & 1;
      if (!mbar_wait_warp(smem_u32(&full_bar[s]), ph, status, 32)) break;
      tcgen05_fence_after();
      if (elected) {
        const uint32_t a = smem_u32(smem + s * C::kStage), b = a + C::kStageA;
#pragma unroll
        for (int k = 0; k < kRgK / 16; ++k)       // 16 elements are 32 bytes further along the swizzled rows
          tcgen05_mma_f16(tmem, desc_kmajor<128>(a + 32 * k), desc_kmajor<128>(b + 32 * k), idesc, (i > 0 || k > 0) ? 1u : 0u);
        tcgen05_commit(smem_u32(&empty_bar[s]));
        if (i == n_steps - 1) tcgen05_commit(smem_u32(acc_full));
      }
      __syncwarp();
    }
  } else {
    bool ok = mbar_wait(smem_u32(acc_full), 0, status, 33);
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
      tcgen05_fence_after();
      const int quarter = warp & 3;               // tensor-memory lanes [32 quarter, +32) belong to this warp
      const int m = m0 + quarter * 32 + lane;
      float* dst = parts + ((int64_t)blockIdx.z * M + m) * E + e0;
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t r[32];
        tcgen05_ld_32x32(tmem + ((uint32_t)(quarter * 32) << 16) + c * 32, r);
        tcgen05_wait_ld();
        const int left = E - e0 - c * 32;
        if (m < M && left > 0) {
          if (left >= 32 && (E & 3) == 0 && (reinterpret_cast<uintptr_t>(parts) & 15) == 0) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
              reinterpret_cast<uint4*>(dst + c * 32)[i] = make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (i < left) dst[c * 32 + i] = __uint_as_float(r[i]);
          }
        }
      }
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)BN) : "memory");
  }
}

// ------------------------------------------------------------------------------------------ top-k

// unsigned keys in the order of the floats; 0 is below every float
__device__ __forceinline__ uint32_t float_key(float v) {
  const uint32_t u = __float_as_uint(v);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_float(uint32_t k) { return __uint_as_float((k & 0x80000000u) ? (k ^ 0x80000000u) : ~k); }

// The k largest of the 32 * PER keys of a warp (lane-interleaved: expert e in lane e % 32, slot e / 32) for one token, and their weights.
// The arg-max of a round is two warp reductions (largest key, then the lowest expert id that holds it); shuffle trees of
// (value, id) pairs over 32 slots per lane took 5.8 us at M=32.
template <int PER>
__device__ __forceinline__ void select_topk(uint32_t (&key)[PER], int lane, int topk, int renormalize, float* topk_w, int32_t* topk_ids) {
  float mx = 0.f, total = 0.f, sel_sum = 0.f, my_w = 0.f;
  int my_id = 0;
  for (int r = 0; r < topk; ++r) {
    uint32_t best = key[0];
#pragma unroll
    for (int i = 1; i < PER; ++i) best = max(best, key[i]);
    const uint32_t top = __reduce_max_sync(0xffffffffu, best);
    uint32_t id = 0xffffffffu;                     // the lane's lowest expert that holds the largest key
#pragma unroll
    for (int i = PER - 1; i >= 0; --i)
      if (key[i] == top) id = i * 32 + lane;
    id = __reduce_min_sync(0xffffffffu, id);
#pragma unroll
    for (int i = 0; i < PER; ++i)                  // compile-time indexed: keeps key[] in registers
      if (id == (uint32_t)(i * 32 + lane)) key[i] = 0u;
    const float value = key_float(top);
    if (r == 0) {
      mx = value;
      if (!renormalize) {
#pragma unroll
        for (int i = 0; i < PER; ++i) total += key[i] != 0u ? __expf(key_float(key[i]) - mx) : 0.f;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) total += __shfl_xor_sync(0xffffffffu, total, d);
        total += 1.f;                              // the largest itself, already taken out
      }
    }
    const float w = __expf(value - mx);
    sel_sum += w;
    if (lane == r) {
      my_w = w;
      my_id = (int)id;
    }
  }
  const float denom = renormalize ? sel_sum : total;
  if (lane < topk) {
    topk_w[lane] = my_w / denom;
    topk_ids[lane] = my_id;
  }
}

// One warp per token; E <= 32 * PER.
template <int PER>
__global__ void __launch_bounds__(128)
    router_topk_kernel(const float* __restrict__ parts, int splits, int M, int E, int topk, int renormalize,
                       float* __restrict__ topk_w, int32_t* __restrict__ topk_ids) {
  pdl_wait();
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31;
  const int m = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (m >= M) return;
  uint32_t key[PER];
  {
    float v[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) v[i] = 0.f;
    for (int z = 0; z < splits; ++z) {
      const float* src = parts + ((int64_t)z * M + m) * E + lane;
#pragma unroll
      for (int i = 0; i < PER; ++i)                // lane-interleaved: expert e lives in lane e % 32, slot e / 32
        if (i * 32 + lane < E) v[i] += src[i * 32];
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) key[i] = i * 32 + lane < E ? float_key(v[i]) : 0u;
  }
  select_topk<PER>(key, lane, topk, renormalize, topk_w + (int64_t)m * topk, topk_ids + (int64_t)m * topk);
}

// Projection, exchange and selection in one launch.  A cluster of CL blocks takes eight tokens: block r the experts
// [16 r tiles, +16 tiles), its warps the 16-expert tiles times slices of K.  In a 32-wide step lane (g, t) = (lane / 4, lane % 4) loads the
// 8 elements at k = 8t of rows g and g + 8 (experts) and g (tokens): the order of k inside a product sum is free, so elements 0-3 of the 8
// serve as the lane's k of one mma and 4-7 as those of another, on both sides alike.  The slices of a logit are added in a fixed order; logits
// go through distributed shared memory to the block that selects for their token: nothing is written to memory but the result.
// Bound by latency (launch, rounds of loads, exchange, selection) and by what one SM reads of the gate through L2.
template <typename T, int CL, int PER>
__global__ void __launch_bounds__(kRcThreads, 1)
    router_cluster_kernel(const T* __restrict__ hidden, int64_t ld_h, const T* __restrict__ gate_w, int M, int H, int E, int tiles, int topk,
                          int renormalize, int* __restrict__ status, float* __restrict__ topk_w, int32_t* __restrict__ topk_ids) {
  __shared__ float s_part[kRcWarps][16][9];       // [slice of K and tile][expert][token]
  __shared__ float s_logit[32 * PER];                      // this block's token, all experts
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int rank = (int)(blockIdx.x % CL), m0 = (int)(blockIdx.x / CL) * 8;
  const int slices = kRcWarps / tiles, tile = warp % tiles, slice = warp / tiles, e_block = rank * tiles * 16, e0 = e_block + tile * 16;
  cluster_sync_any();                                      // the other blocks run before anything is sent to them
  pdl_wait();
  pdl_launch_dependents();
  if (blockIdx.x == 0 && threadIdx.x == 0) *status = 0;
  if (slice < slices) {
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    const T* wa = gate_w + (int64_t)min(e0 + g, E - 1) * H;            // rows past the end repeat the last: never used
    const T* wb = gate_w + (int64_t)min(e0 + g + 8, E - 1) * H;
    const T* x = hidden + (int64_t)min(m0 + g, M - 1) * ld_h;
    const uint4 zero = make_uint4(0, 0, 0, 0);
    constexpr int U = 4;                                   // 32-wide steps in flight
    for (int k0 = 32 * slice; k0 < H; k0 += 32 * U * slices) {
      uint4 a[U][2], b[U];
#pragma unroll
      for (int s = 0; s < U; ++s) {
        const int k = k0 + 32 * slices * s + 8 * t;
        const bool in = k < H;
        a[s][0] = in ? ldg_stream_u4(wa + k) : zero;
        a[s][1] = in ? ldg_stream_u4(wb + k) : zero;
        b[s] = in ? *reinterpret_cast<const uint4*>(x + k) : zero;
      }
#pragma unroll
      for (int s = 0; s < U; ++s) {
        mma_m16n8k16<T>(acc, a[s][0].x, a[s][1].x, a[s][0].y, a[s][1].y, b[s].x, b[s].y);
        mma_m16n8k16<T>(acc, a[s][0].z, a[s][1].z, a[s][0].w, a[s][1].w, b[s].z, b[s].w);
      }
    }
    s_part[warp][g][2 * t] = acc[0];
    s_part[warp][g][2 * t + 1] = acc[1];
    s_part[warp][g + 8][2 * t] = acc[2];
    s_part[warp][g + 8][2 * t + 1] = acc[3];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < tiles * 16 * 8; i += kRcThreads) {
    const int e = i % (tiles * 16), tok = i / (tiles * 16);
    float v = 0.f;
    for (int z = 0; z < slices; ++z) v += s_part[z * tiles + (e >> 4)][e & 15][tok];
    if (e_block + e < E) {
      const uint32_t to = map_to_cta(smem_u32(&s_logit[e_block + e]), (uint32_t)tok);
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(to), "f"(v) : "memory");
    }
  }
  cluster_sync_any();
  const int m = m0 + rank;
  if (warp == 0 && rank < 8 && m < M) {
    uint32_t key[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) key[i] = i * 32 + lane < E ? float_key(s_logit[i * 32 + lane]) : 0u;
    select_topk<PER>(key, lane, topk, renormalize, topk_w + (int64_t)m * topk, topk_ids + (int64_t)m * topk);
  }
}

// ------------------------------------------------------------------------------------------ host

// Which way a call goes.  One launch of clusters saves a launch, but only 8 or 16 SMs read the gate for eight tokens, and those without experts
// none of it.  In a graph only the GPU's time counts (us, clusters / slices and selection):
//   M=8: 32 experts H=2048 3.9 / 3.3, H=12800 8.8 / 5.0   64, 3072 4.5 / 3.8   128, 7168 6.3 / 5.3   512, 7168 9.8 / 7.4
//   M=16: 32, 2048 3.9 / 3.6   64, 3072 4.5 / 4.2   128, 7168 6.4 / 5.7   512, 9216 11.7 / 9.0
// Called one by one, two launches take the host about 7 us, whatever they are, one 4.4: clusters as far as they take less than that (from Python):
//   M=8: 32, 2048 4.4 / 7.3, H=9216 6.6 / 7.2, H=10240 6.9 / 7.2, H=12800 8.2 / 7.1   128, 7168 5.8 / 7.3, H=10240 7.0 / 7.0, H=12800 8.3 / 7.0
//   M=16: 64, 9216 6.9 / 6.8, H=10240 7.1 / 6.9, H=12800 8.4 / 6.9   512 (M=8), 7168 9.3 / 7.4, H=9216 11.1 / 8.0
// From 17 tokens on clusters are the faster ones up to 512 experts; the tiles read the whole gate once for 128 tokens, the slices once for 8 to 32
// (slices / tiles; M=17: 1000 experts H=2048 10.9 / 13.1, H=4096 13.3 / 14.1, H=7168 18.5 / 15.8; M=64, H=4096 19.4 / 15.2; M=8, H=12800 20.8 / 19.4).
constexpr int kRtClusterMaxTokens = 64;
constexpr int kRtSlicesMaxTokens = 32;
constexpr int kRtMaxSplits = 8;

enum class RouterPath { kClusters, kSlices, kTiles };

RouterPath router_path(int64_t M, int64_t H, int64_t E, cudaStream_t st) {
  const int64_t gate = E * H;
  if (M <= 16) {
    if (E <= 128)
      return H > 10240 || (H > (E <= 32 ? 1536 : E <= 64 ? 2560 : 6144) && stream_capturing(st)) ? RouterPath::kSlices : RouterPath::kClusters;
    if (gate <= (M <= 8 ? 3200000 : 3900000)) return RouterPath::kClusters;
    return E <= 512 || gate <= (M <= 8 ? 9300000 : 7500000) ? RouterPath::kSlices : RouterPath::kTiles;
  }
  if (E <= 512) return M <= kRtClusterMaxTokens ? RouterPath::kClusters : RouterPath::kTiles;
  return M <= kRtSlicesMaxTokens && H <= (E > 896 ? 4608 : 3072) ? RouterPath::kSlices : RouterPath::kTiles;
}

// K-slices of the projection: enough blocks to cover the SMs, at most eight (the top-k kernel reads them all)
int router_splits(int64_t blocks) {
  const int64_t z = sm_count() / (blocks > 0 ? blocks : 1);
  return (int)(z < 1 ? 1 : (z > kRtMaxSplits ? kRtMaxSplits : z));
}
int slices_splits(int64_t E) { return router_splits((E + 15) / 16); }       // one block of tokens

struct TileShape {
  int bn, splits;
};
TileShape tile_shape(int64_t M, int64_t E) {
  TileShape s;
  const int64_t mt = (M + 127) / 128;
  s.bn = mt * ((E + 127) / 128) <= sm_count() ? 128 : 256;
  s.splits = router_splits(mt * ((E + s.bn - 1) / s.bn));
  return s;
}

template <typename T>
void launch_router_slices(int splits, const void* hidden, int64_t ld_h, const void* gate_w, int M, int H, int E, int* status, float* parts,
                          cudaStream_t st) {
  auto go = [&](auto kernel) {
    launch_pdl(kernel, dim3((unsigned)((E + 15) / 16), 1, (unsigned)splits), dim3(kRsThreads), 0, st, static_cast<const T*>(hidden), ld_h,
               static_cast<const T*>(gate_w), M, H, E, status, parts);
  };
  if (M <= 8) go(router_slices_kernel<T, 1>);
  else if (M <= 16) go(router_slices_kernel<T, 2>);
  else go(router_slices_kernel<T, 4>);
}

template <typename T, int CL, int PER>
int resident_router_clusters() {
  static ResidentClusters counts[64];
  return resident_clusters_of(counts, router_cluster_kernel<T, CL, PER>, CL, kRcThreads, 0);
}

template <typename T, int CL, int PER>
cudaError_t launch_router_cluster_t(const void* hidden, int64_t ld_h, const void* gate_w, int M, int H, int E, int topk, int renormalize,
                                    int* status, float* topk_w, int32_t* topk_ids, cudaStream_t st) {
  const int tiles = (E + 16 * CL - 1) / (16 * CL);
  return launch_pdl_cluster(CL, router_cluster_kernel<T, CL, PER>, dim3((unsigned)(CL * ((M + 7) / 8))), dim3(kRcThreads), 0, st,
                            static_cast<const T*>(hidden), ld_h, static_cast<const T*>(gate_w), M, H, E, tiles, topk, renormalize, status,
                            topk_w, topk_ids);
}

// Sixteen blocks to a cluster where there are experts for them and all clusters run at once (512 experts, H=2048, us with 8 / 16: M=1 6.5 / 4.8,
// M=32 7.6 / 5.6, M=64 7.4 / 10.5 with an eighth cluster that waits; 256 experts, M=32 4.8 / 4.0), else eight.
template <typename T>
int launch_router_cluster(const void* hidden, int64_t ld_h, const void* gate_w, int M, int H, int E, int topk, int renormalize, int* status,
                          float* topk_w, int32_t* topk_ids, cudaStream_t st) {
  auto go = [&](auto* launch) { return launch(hidden, ld_h, gate_w, M, H, E, topk, renormalize, status, topk_w, topk_ids, st); };
  const int clusters = (M + 7) / 8;
  cudaError_t rc;
  if (E <= 128) rc = go(launch_router_cluster_t<T, 8, 4>);
  else if (E <= 256) rc = clusters <= resident_router_clusters<T, 16, 8>() ? go(launch_router_cluster_t<T, 16, 8>) : go(launch_router_cluster_t<T, 8, 8>);
  else if (E > 512) rc = resident_router_clusters<T, 16, kRtPerLane>() > 0 ? go(launch_router_cluster_t<T, 16, kRtPerLane>) : go(launch_router_cluster_t<T, 8, kRtPerLane>);
  else rc = clusters <= resident_router_clusters<T, 16, 16>() ? go(launch_router_cluster_t<T, 16, 16>) : go(launch_router_cluster_t<T, 8, 16>);
  if (rc != cudaSuccess) {
    cudaGetLastError();
    return B200FP4_STATUS_EXECUTION_FAILED;
  }
  return finish_launch(1);
}

template <int BN>
int launch_router_gemm(const CUtensorMap& mx, const CUtensorMap& mw, int splits, bool bf16, int M, int H, int E, int* status,
                       float* parts, cudaStream_t st) {
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return B200FP4_STATUS_NOT_SUPPORTED;
  if (!attr_set[dev]) {
    if (cudaFuncSetAttribute(router_gemm_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RouterGemm<BN>::kSmem) != cudaSuccess) {
      cudaGetLastError();
      return B200FP4_STATUS_EXECUTION_FAILED;
    }
    attr_set[dev] = true;
  }
  const uint32_t fmt = bf16 ? 1u : 0u;        // fp32 accumulators, f16 / bf16 operands, K-major both, N = BN, M = 128
  const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(BN >> 3) << 17) | ((128u >> 4) << 24);
  const dim3 grid((unsigned)((E + BN - 1) / BN), (unsigned)((M + 127) / 128), (unsigned)splits);
  launch_pdl(router_gemm_kernel<BN>, grid, dim3(kRgThreads), RouterGemm<BN>::kSmem, st, mx, mw, M, H, E, idesc, status, parts);
  return B200FP4_STATUS_SUCCESS;
}

}  // namespace
}  // namespace b200fp4

using namespace b200fp4;

// workspace: 256 bytes (first int: status word of the tcgen05 kernel's bounded waits), then the K-slices of the logits.  Enough for whichever
// path the width of the gate leads to, and up to 128 tokens for every smaller batch too.
extern "C" size_t b200fp4_moe_router_workspace_bytes(int64_t M, int64_t E) {
  if (M <= 0 || E <= 0) return 0;
  const int64_t tiles = M > kRtClusterMaxTokens || E > 512 ? tile_shape(M, E).splits * M : 0;
  const int64_t slices = slices_splits(E) * (M < kRtSlicesMaxTokens ? M : (int64_t)kRtSlicesMaxTokens);
  return 256 + (size_t)(tiles > slices ? tiles : slices) * (size_t)E * sizeof(float);
}

extern "C" int b200fp4_moe_router(const void* hidden, int64_t ld_h, int dtype, const void* gate_w, int64_t M, int64_t H,
                                  int64_t E, int64_t topk, int renormalize, float* topk_weights, int32_t* topk_ids,
                                  void* workspace, size_t workspace_bytes, void* stream) {
  if (M < 0 || H <= 0 || E <= 0 || topk <= 0 || (H % 8) != 0 || ld_h < H || (ld_h % 8) != 0) return B200FP4_STATUS_INVALID_VALUE;
  if (dtype != B200FP4_DTYPE_BF16 && dtype != B200FP4_DTYPE_F16) return B200FP4_STATUS_NOT_SUPPORTED;
  if (topk > 32 || topk > E || E > 32 * kRtPerLane || H > 12800) return B200FP4_STATUS_NOT_SUPPORTED;
  if (M == 0) return B200FP4_STATUS_SUCCESS;
  if (!hidden || !gate_w || !topk_weights || !topk_ids || !aligned(hidden, 16) || !aligned(gate_w, 16))
    return B200FP4_STATUS_INVALID_VALUE;
  cudaStream_t st = (cudaStream_t)stream;
  const RouterPath path = router_path(M, H, E, st);
  const size_t need = path == RouterPath::kClusters ? 256 : b200fp4_moe_router_workspace_bytes(M, E);      // clusters keep their logits on chip
  if (!workspace || workspace_bytes < need || !aligned(workspace, 4)) return B200FP4_STATUS_ALLOC_FAILED;
  if (M > (int64_t)65535 * 128) return B200FP4_STATUS_NOT_SUPPORTED;
  int* status = static_cast<int*>(workspace);
  float* parts = reinterpret_cast<float*>(static_cast<unsigned char*>(workspace) + 256);
  const bool bf = dtype == B200FP4_DTYPE_BF16;
  int splits;
  if (path == RouterPath::kClusters) {
    auto* go = bf ? launch_router_cluster<__nv_bfloat16> : launch_router_cluster<__half>;
    return go(hidden, ld_h, gate_w, (int)M, (int)H, (int)E, (int)topk, renormalize, status, topk_weights, topk_ids, st);
  } else if (path == RouterPath::kSlices) {
    splits = slices_splits(E);
    const int most = (int)((H + 64 * kRsWarps - 1) / (64 * kRsWarps));       // no more slices than there are rounds of 64 per warp
    if (splits > most) splits = most;
    auto* go = bf ? launch_router_slices<__nv_bfloat16> : launch_router_slices<__half>;
    go(splits, hidden, ld_h, gate_w, (int)M, (int)H, (int)E, status, parts, st);
  } else {
    const TileShape sh = tile_shape(M, E);
    splits = sh.splits;
    if (b200fp4_has_hardware_acceleration() != 1) return B200FP4_STATUS_ARCH_MISMATCH;
    const int most = (int)((H + 4 * kRgK - 1) / (4 * kRgK));       // at least about four stages per slice
    if (splits > most) splits = most;
    CUtensorMap mx, mw;
    if (!make_rows_map(&mx, hidden, (uint64_t)M, (uint64_t)H * 2, (uint64_t)ld_h * 2, 128, 128) ||
        !make_rows_map(&mw, gate_w, (uint64_t)E, (uint64_t)H * 2, (uint64_t)H * 2, (uint32_t)sh.bn, 128))
      return B200FP4_STATUS_INTERNAL_ERROR;
    const int rc = sh.bn == 128 ? launch_router_gemm<128>(mx, mw, splits, bf, (int)M, (int)H, (int)E, status, parts, st)
                                : launch_router_gemm<256>(mx, mw, splits, bf, (int)M, (int)H, (int)E, status, parts, st);
    if (rc != B200FP4_STATUS_SUCCESS) return rc;
  }
  auto topk_go = [&](auto kernel) {
    launch_pdl(kernel, dim3((unsigned)((M + 3) / 4)), dim3(128), 0, st, (const float*)parts, splits, (int)M, (int)E, (int)topk,
               renormalize, topk_weights, topk_ids);
  };
  if (E <= 64) topk_go(router_topk_kernel<2>);
  else if (E <= 128) topk_go(router_topk_kernel<4>);
  else if (E <= 256) topk_go(router_topk_kernel<8>);
  else if (E <= 512) topk_go(router_topk_kernel<16>);
  else topk_go(router_topk_kernel<kRtPerLane>);
  return finish_launch(2);
}
