// NVFP4 linear layer / GEMM of few tokens for sm_100a: out[M,N] = alpha * (A . sfA)(B . sfB)^T, M <= kSmallMaxM.
//
// A decode step's linear layer reads its weight once for a few tokens, so what counts is how soon the weight is requested, how
// many SMs request it, and the launches.  Against the general kernel (gemm.cu) here
//   * the operands change places: the 128 rows of an MMA are rows of the WEIGHT and the tokens are its 8..64 columns, so that
//     nothing is computed, loaded or kept in tensor memory for padding rows (a tile of 128 tokens has 120 of them at M = 8);
//   * the activations are quantized by the kernel itself, each CTA its own part of K for all tokens, straight into the operand's
//     shared-memory layout while the first weight tiles are on their way: one launch instead of two, no trip of codes and scales
//     through memory.  The arithmetic is the quantizer's (quant.cuh), the bytes are the same;
//   * K is split over clusters of up to eight CTAs, whatever number fits the SMs; the partial sums of a token go through distributed
//     shared memory, each of its four 32-column pieces to another CTA of the cluster, and are added there in the order of K.
// The GEMM on codes that are already there (cutlass_scaled_fp4_mm) takes the same kernel where that is the faster one, with the quantization
// replaced by a copy.
// What bounds it: the chain of copy, quantization, scales, MMA, exchange and store where the weight is small, HBM where it is large.
// Measured back to back (us; quantizer and general kernel / so): M=8 N=512 K=2048 7.1 / 4.1, M=1 N=K=4096 8.9 / 6.1, M=1 N=14336
// K=4096 14.0 / 8.9 (3.8 TB/s), M=16 of that 13.5 / 12.0, M=24 N=1536 K=3008 7.8 / 6.4.  Weight scales take about as long to reach tensor memory as a
// stage takes to arrive, which is why two stages share a wait there.
// One tile per CTA.  Warps: 0 copies of the weight and its scales, 1 MMA, 2-5 the weight's and 6-9 the activations' scale factors into
// tensor memory, all eight the epilogue, 10-25 activations.  Every mbarrier wait is bounded (status word), tensor memory is always freed.
#include <type_traits>

#include "gemm_small.cuh"
#include "quant.cuh"
#include "sm100_ptx.cuh"

namespace b200fp4 {
namespace {

constexpr int kXWarps = 16;                    // warps that bring the activations in
constexpr int kFirstXWarp = 10;
constexpr int kThreads = 32 * (kFirstXWarp + kXWarps);
constexpr int kRingMost = 8;                   // weight stages: 128 rows x 256 k of codes and their scales
constexpr int kStageA = 128 * 128, kStageSfa = 4 * 512;
constexpr int kMaxStages = 32;                 // 256-wide stages of K one CTA may own
constexpr int kMaxSplit = 8;
constexpr size_t kSmemMost = 227 * 1024;

struct SmallParams {
  const void* x;              // [M, K] 16-bit activations, rows ldx elements apart; or packed codes [M, K/2]
  int64_t ldx;
  const float* gs;            // activations' global scale (16-bit input only)
  const uint8_t* x_sf;        // swizzled scales of given codes
  const uint8_t* w_sf;        // swizzled scales of the weight
  const float* alpha;
  void* out;
  int out_dtype;
  int load32;                 // rows of x are 32-byte aligned
  int M, N, K;
  int m_pad;                  // columns of an MMA: M rounded up to a multiple of 8
  int split, stages, ring;    // CTAs per tile, 256-wide stages of the whole K, weight stages in flight
  int warps_per_stage;        // activation warps that share a stage
  uint32_t tmem_cols;
  int* status;
};

// Shared memory behind the 1024-byte aligned base: weight ring | weight scales | activation codes [stage][m_pad rows of 128 bytes,
// swizzled] | activation scales [64 of k][32-token group][token][4] | partial sums [source CTA][owned token][128] | table of
// quantizer multipliers | barriers
struct Layout {
  uint32_t sfa, xq, xsf, part, table, bars, bytes;
};
__host__ __device__ __forceinline__ Layout small_layout(int ring, int own_stages, int m_pad, int M, int split) {
  Layout l;
  l.sfa = (uint32_t)ring * kStageA;
  l.xq = l.sfa + (uint32_t)ring * kStageSfa;
  l.xsf = l.xq + (uint32_t)own_stages * m_pad * 128;
  l.part = l.xsf + (uint32_t)own_stages * 4 * ((m_pad + 31) / 32) * 128;
  l.table = l.part + (split > 1 ? (uint32_t)split * ((M + split - 1) / split) * 512 : 0);
  l.bars = l.table + 128 * 4;
  l.bytes = l.bars + (3 * kRingMost + kMaxStages + 2) * 8;
  return l;
}

__device__ __forceinline__ void tcgen05_ld_32x8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}

__device__ __forceinline__ void store_one(const SmallParams& p, int m, int n, float v) {
  const size_t at = (size_t)m * p.N + n;
  if (p.out_dtype == B200FP4_DTYPE_BF16) static_cast<__nv_bfloat16*>(p.out)[at] = __float2bfloat16_rn(v);
  else if (p.out_dtype == B200FP4_DTYPE_F16) static_cast<__half*>(p.out)[at] = __float2half_rn(v);
  else static_cast<float*>(p.out)[at] = v;
}

// T: type of the activations; kCodes: they are packed codes with swizzled scales already
template <typename T, bool kCodes>
__global__ void __launch_bounds__(kThreads, 1)
    nvfp4_small_kernel(const __grid_constant__ CUtensorMap map_w, const SmallParams p) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)(blockIdx.x % (unsigned)p.split), tile = (int)(blockIdx.x / (unsigned)p.split);
  const int ks_begin = p.stages * rank / p.split, n_ks = p.stages * (rank + 1) / p.split - ks_begin;      // this CTA's part of K
  const int most_ks = (p.stages + p.split - 1) / p.split, ring = p.ring, M = p.M, m_pad = p.m_pad, words = (m_pad + 31) >> 5;
  const Layout L = small_layout(ring, most_ks, m_pad, M, p.split);
  const uint32_t base = smem_u32(smem);
  const uint32_t full_bar = base + L.bars, empty_bar = full_bar + 8 * kRingMost, sf_full = empty_bar + 8 * kRingMost;
  const uint32_t x_full = sf_full + 8 * kRingMost;
  const uint32_t acc_full = x_full + 8 * kMaxStages, tmem_ptr = acc_full + 8;
  int* const status = p.status;
  if (threadIdx.x == 0) {
    for (int s = 0; s < ring; ++s) {
      mbar_init(full_bar + 8 * s, 9);              // the weight tile, and each scale-factor warp
      mbar_init(empty_bar + 8 * s, 1);
      mbar_init(sf_full + 8 * s, 1);
    }
    for (int i = 0; i < n_ks; ++i) mbar_init(x_full + 8 * i, p.warps_per_stage);
    mbar_init(acc_full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_ptr), "r"(p.tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  if (p.split > 1) cluster_sync_any();             // the other CTAs run before anything is sent to them
  else __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = lds32(tmem_ptr);
  const uint32_t tmem_sf = tmem + ((m_pad + 31) & ~31);          // 32 columns per weight stage: 16 weight, 16 activations
  const int KT = p.K >> 6;                         // 64-wide k-blocks
  // The arguments are fetched here, while the kernel before this one ends: a first read of them further down waits for the
  // constant cache with the weight not yet requested.
  asm volatile("" ::"l"(p.x), "l"(p.ldx), "l"(p.gs), "l"(p.x_sf), "l"(p.w_sf), "l"(p.alpha), "l"(p.out), "r"(p.out_dtype), "r"(p.load32),
               "r"(p.N), "r"(p.split), "l"(status));
  pdl_wait();
  const float alpha = *p.alpha;

  if (warp == 0) {
    // ------------------------------------------------------------------ copies of the weight and its scales
    const bool leader = elect_one();
    const uint8_t* sf = p.w_sf + ((size_t)tile * KT + (size_t)ks_begin * 4) * 512;
    int s = 0;
    uint32_t ph = 1;
    for (int i = 0; i < n_ks; ++i, sf += kStageSfa) {
      if (i >= ring && !mbar_wait_warp(empty_bar + 8 * s, ph, status, 41)) break;
      if (leader) {
        const uint32_t bar = full_bar + 8 * s, sbar = sf_full + 8 * s, sf_bytes = (uint32_t)min(4, KT - (ks_begin + i) * 4) * 512;
        mbar_expect_tx(bar, kStageA);
        tma_load_2d(base + s * kStageA, &map_w, (ks_begin + i) * 128, tile * 128, bar);
        mbar_expect_tx(sbar, sf_bytes);
        bulk_load_1d(base + L.sfa + s * kStageSfa, sf, sf_bytes, sbar);
      }
      __syncwarp();
      if (++s == ring) {
        s = 0;
        ph ^= 1;
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    // E2M1 x E2M1, UE4M3 scales, K-major A and B, M = 128, N = m_pad, K = 64
    const bool leader = elect_one();
    const uint32_t idesc = (1u << 7) | (1u << 10) | ((uint32_t)(m_pad >> 3) << 17) | (8u << 24);
    const uint64_t a0 = desc_kmajor<128>(base), b0 = desc_kmajor<128>(base + L.xq);
    bool ok = true;
    int s = 0;
    uint32_t ph = 0;
    for (int i = 0; i < n_ks; ++i) {
      ok = mbar_wait_warp(full_bar + 8 * s, ph, status, 42);
      if (!ok) break;
      tcgen05_fence_after();
      if (leader) {
        const uint64_t a = a0 + s * (kStageA >> 4), b = b0 + (uint64_t)((uint32_t)i * m_pad * 8);
        const uint32_t sfa = tmem_sf + s * 32, sfb = sfa + 16;
        const int kblocks = KT - (ks_begin + i) * 4;
#pragma unroll
        for (int kb = 0; kb < 4; ++kb)             // 64 of k are 32 bytes further along the swizzled rows
          if (kb < kblocks) tcgen05_mma_nvf4(tmem, a + kb * 2, b + kb * 2, idesc, sfa + kb * 4, sfb + kb * 4, (i > 0 || kb > 0) ? 1u : 0u);
        if (i + ring < n_ks) tcgen05_commit(empty_bar + 8 * s);
        if (i == n_ks - 1) tcgen05_commit(acc_full);
      }
      __syncwarp();
      if (++s == ring) {
        s = 0;
        ph ^= 1;
      }
    }
  } else if (warp < kFirstXWarp) {
    // ------------------------------------------------------------------ scale factors, then the epilogue
    // Lane L of each 32-lane quarter of tensor memory holds the scales of rows L, L + 32, L + 64, L + 96: a word per row and
    // 64-wide k-block, the four quarters alike.  Stages of fewer than four k-blocks copy what lies behind: no MMA reads it.
    const int quarter = warp & 3;
    const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
    bool ok = true;
    int s = 0;
    uint32_t ph = 0;
    for (int i = 0; i < n_ks; i += 2) {
      // two stages per turn: the wait for the stores to tensor memory, most of a turn, is paid once for both
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int t = s + j == ring ? 0 : s + j;
        const uint32_t pt = s + j == ring ? ph ^ 1 : ph;
        if (!ok || i + j >= n_ks) break;
        uint4 w[4];
        if (warp < 6) {
          // the copies into a slot wait for the MMAs that have read it, and so does this
          ok = __all_sync(0xffffffffu, mbar_wait(sf_full + 8 * t, pt, status, 43));
          if (!ok) break;
          const uint32_t src = base + L.sfa + t * kStageSfa + lane * 16;
#pragma unroll
          for (int kb = 0; kb < 4; ++kb) w[kb] = lds128(src + kb * 512);
        } else {
          ok = __all_sync(0xffffffffu, (i + j < ring || mbar_wait(empty_bar + 8 * t, pt ^ 1, status, 44)) &&
                                           mbar_wait(x_full + 8 * (i + j), 0, status, 45));
          if (!ok) break;
          // rows past M: zero, whatever their codes are
          const uint32_t src = base + L.xsf + (uint32_t)(i + j) * 4 * words * 128 + lane * 4;
#pragma unroll
          for (int kb = 0; kb < 4; ++kb)
            w[kb] = make_uint4(lane < M ? lds32(src + kb * words * 128) : 0u, lane + 32 < M ? lds32(src + (kb * words + 1) * 128) : 0u, 0u, 0u);
        }
        tcgen05_fence_after();                     // the slot's columns were read by MMAs whose commit these waits follow
        const uint32_t t0 = tmem_sf + lanes + t * 32 + (warp < 6 ? 0 : 16);
#pragma unroll
        for (int kb = 0; kb < 4; ++kb) tcgen05_st_32x32_x4(t0 + kb * 4, w[kb]);
      }
      if (!ok) break;
      tcgen05_wait_st();
      tcgen05_fence_before();
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (i + j < n_ks && lane == 0) mbar_arrive(full_bar + 8 * s);
        if (++s == ring) {
          s = 0;
          ph ^= 1;
        }
      }
    }
    if (ok) ok = __all_sync(0xffffffffu, mbar_wait(acc_full, 0, status, 46));
    if (ok) {
      // tensor-memory lane = output column, tensor-memory column = token: a warp writes 32 neighbouring outputs of a token at once
      tcgen05_fence_after();
      const int n = tile * 128 + quarter * 32 + lane, split = p.split;
      const int owned = (M + split - 1) / split;
      for (int c = warp < 6 ? 0 : 8; c < m_pad; c += 16) {
        uint32_t r[8];
        tcgen05_ld_32x8(tmem + lanes + c, r);
        tcgen05_wait_ld();
        if (split == 1) {
          if (n < p.N) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (c + j < M) store_one(p, c + j, n, __uint_as_float(r[j]) * alpha);
          }
          continue;
        }
        // the 32 outputs of token m are finished by CTA (m + quarter) % split, so that the warps of a CTA send to different CTAs
        // at any time: [sender][m / split][column]
        int idx = c / split, rem = c - idx * split;
        uint32_t owner = (uint32_t)(rem + quarter) % (uint32_t)split;
        uint32_t to = base + L.part + ((uint32_t)(rank * owned + idx) * 128 + quarter * 32 + lane) * 4;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (c + j < M)
            asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(map_to_cta(to, owner)), "r"(r[j]) : "memory");
          if (++owner == (uint32_t)split) owner = 0;
          if (++rem == split) {
            rem = 0;
            to += 512;
          }
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ activations
    // Groups of warps_per_stage warps take stages in turn; a thread has up to four blocks of 16 of a stage in flight.
    const int wps = p.warps_per_stage, xw = warp - kFirstXWarp, groups = kXWarps / wps, group = xw / wps;
    const int first = (xw - group * wps) * 32 + lane, step = wps * 32;
    const int units = M * 16, KB = p.K >> 4;
    const float* table = reinterpret_cast<const float*>(smem + L.table);
    // A negative global scale gives every scale byte its sign and the codes of its magnitude: 1 / (decoded scale / global scale) is the same.
    const float given_gs = kCodes ? 0.f : p.gs[0], gs = fabsf(given_gs);
    const uint32_t sf_sign = (__float_as_uint(given_gs) >> 31) << 7;
    bool table_made = false;
    // The multiplier of every scale byte, made while the first loads are on their way: with it a block's chain of dependent
    // operations is two reciprocals shorter.
    auto make_table = [&]() {
      if (kCodes || table_made) return;
      table_made = true;
      const int t = threadIdx.x - 32 * kFirstXWarp;
      if (t < 128) {
        const float rcp_gs = __frcp_rn(gs + (gs == 0.f ? 1.0e8f : 0.f));
        reinterpret_cast<float*>(smem + L.table)[t] = out_scale_of((uint8_t)t, rcp_gs);
      }
      __syncwarp();
      asm volatile("bar.sync 1, %0;" ::"n"(32 * kXWarps) : "memory");
    };
    auto stages_of = [&](auto blocks) {
      constexpr int B = decltype(blocks)::value;   // in flight per thread
      for (int i = group; i < n_ks; i += groups) {
        const int kb0 = (ks_begin + i) * 16;       // first block of 16 of the stage
        unsigned char* xq = smem + L.xq + (uint32_t)i * m_pad * 128;
        unsigned char* xsf = smem + L.xsf + (uint32_t)i * 4 * words * 128;
        for (int u0 = 0; u0 < units; u0 += B * step) {
          uint4 r0[B], r1[B];
#pragma unroll
          for (int j = 0; j < B; ++j) {
            const int u = u0 + first + j * step, m = u >> 4, kb = kb0 + (u & 15);
            r0[j] = r1[j] = make_uint4(0, 0, 0, 0);
            if (u < units && kb < KB) {
              if constexpr (kCodes) {
                const uint2 c = *reinterpret_cast<const uint2*>(static_cast<const uint8_t*>(p.x) + (size_t)m * (p.K / 2) + kb * 8);
                r0[j].x = c.x;
                r0[j].y = c.y;
                r0[j].z = p.x_sf[sf_swizzled_offset(m, kb, KT)];
              } else {
                const T* src = static_cast<const T*>(p.x) + (int64_t)m * p.ldx + (int64_t)kb * 16;
                if (p.load32) {
                  ldg_stream_v8(src, r0[j], r1[j]);
                } else {
                  r0[j] = ldg_stream_u4(src);
                  r1[j] = ldg_stream_u4(src + 8);
                }
              }
            }
          }
          make_table();
#pragma unroll
          for (int j = 0; j < B; ++j) {
            const int u = u0 + first + j * step, m = u >> 4, kb = u & 15;
            if (u < units) {
              uint32_t sfb = r0[j].z;
              uint2 c = make_uint2(r0[j].x, r0[j].y);
              if constexpr (!kCodes) c = quantize_block16<T>(r0[j], r1[j], gs, [&](uint32_t b) { return table[b & 127]; }, sfb);
              // rows of 128 bytes in atoms of eight, 16-byte chunk k of row r at k ^ (r % 8)
              *reinterpret_cast<uint2*>(xq + (m >> 3) * 1024 + (m & 7) * 128 + (((kb >> 1) ^ (m & 7)) << 4) + (kb & 1) * 8) = c;
              xsf[((kb >> 2) * words + (m >> 5)) * 128 + (m & 31) * 4 + (kb & 3)] = (uint8_t)(sfb | sf_sign);
            }
          }
        }
        fence_proxy_async_smem();                  // the tensor core reads the codes through the async proxy
        __syncwarp();
        if (lane == 0) mbar_arrive(x_full + 8 * i);
      }
    };
    if (units <= step) stages_of(std::integral_constant<int, 1>{});
    else stages_of(std::integral_constant<int, 4>{});
    make_table();                                  // every warp comes to its barrier
    pdl_launch_dependents();
    if (blockIdx.x == 0 && threadIdx.x == kThreads - 1) *status = 0;      // a wait writes it only after ~1 s
  }
  __syncwarp();
  if (p.split > 1) {
    cluster_sync_any();                            // every CTA's sums have arrived (or a wait ran out: the status word says so)
    const int split = p.split, owned = (M + split - 1) / split;
    for (int i = threadIdx.x; i < owned * 128; i += kThreads) {
      const int idx = i >> 7, col = i & 127, n = tile * 128 + col;
      const int m = idx * split + (rank - (col >> 5) + 4 * split) % split;
      if (m < M && n < p.N) {
        const uint32_t src = base + L.part + (uint32_t)i * 4;
        float v[kMaxSplit];
#pragma unroll
        for (int k = 0; k < kMaxSplit; ++k) v[k] = k < split ? __uint_as_float(lds32(src + (uint32_t)(k * owned) * 512)) : 0.f;
        float sum = v[0];
#pragma unroll
        for (int k = 1; k < kMaxSplit; ++k) sum = k < split ? sum + v[k] : sum;      // in the order of K
        store_one(p, m, n, sum * alpha);
      }
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(p.tmem_cols) : "memory");
  }
}

template <typename T, bool kCodes>
int launch_small_t(const CUtensorMap& mw, const SmallParams& p, unsigned grid, size_t smem, cudaStream_t st) {
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return B200FP4_STATUS_NOT_SUPPORTED;
  if (!attr_set[dev]) {
    if (cudaFuncSetAttribute(nvfp4_small_kernel<T, kCodes>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMost) != cudaSuccess) {
      cudaGetLastError();
      return B200FP4_STATUS_EXECUTION_FAILED;
    }
    attr_set[dev] = true;
  }
  if (launch_pdl_cluster(p.split, nvfp4_small_kernel<T, kCodes>, dim3(grid), dim3(kThreads), smem, st, mw, p) != cudaSuccess) {
    cudaGetLastError();
    return B200FP4_STATUS_EXECUTION_FAILED;
  }
  return finish_launch(1);
}

// Clusters of k CTAs (2 to 8) that run at once
int resident_clusters(int k) {
  static ResidentClusters counts[kMaxSplit + 1][64];
  return resident_clusters_of(counts[k], nvfp4_small_kernel<__nv_bfloat16, false>, k, kThreads, kSmemMost);
}

}  // namespace

SmallPlan small_gemm_plan(int64_t M, int64_t N, int64_t K, SmallUse use) {
  SmallPlan s = {};
  const int64_t sms = sm_count(), tiles = (N + 127) / 128, stages = (K + 255) / 256;
  if (M < 1 || M > kSmallMaxM || tiles > sms) return s;
  // As many CTAs per tile as the chip holds at once: clusters lie within a GPC and leave some of its SMs unused (of 148, 15 clusters of
  // eight; a 16th waits for the others: M=33, N=K=2048 11.8 us, 7.2 so).  Fewer than four stages are not split.
  int split = 1;
  for (int k = 2; k <= kMaxSplit && stages >= 4 && k <= stages; ++k)
    if (tiles * k <= sms && tiles <= resident_clusters(k)) split = k;
  const int own = (int)((stages + split - 1) / split), m_pad = (int)(M + 7) / 8 * 8;
  if (own > kMaxStages) return s;
  // Every CTA brings in its part of K for all tokens and sends its 128 columns out token by token, some 70 cycles a token, where the general path
  // quantizes once and stores tiles; and clusters that nearly fill the chip leave the next launch no room to start in.  So the number of tokens
  // up to which this kernel is the faster one falls with the stages a CTA owns and with the CTAs.  Called one by one, the two launches of the
  // general path take the host at least 6.5 us, so that it reaches further there than in a graph.  Linear, us (quantizer and general kernel /
  // so), from Python and from a graph:
  //   N=K=512 M=45 6.6 / 5.7, 6.5 / 7.0, M=64 6.5 / 6.4, 6.5 / 7.8           N=4096 K=512 M=48 6.7 / 6.0, 6.5 / 7.2, M=64 6.5 / 6.7, 6.7 / 8.0
  //   N=2048 K=1536 M=33 7.1 / 6.4, 7.9 / 7.3   N=1536 K=2048 M=40 7.1 / 6.5, 7.7 / 7.4   N=K=2048 M=48 7.1 / 7.6, 7.7 / 8.5
  //   N=1624 K=2240 M=54 8.2 / 8.0, 9.4 / 8.8   N=1664 K=3072 M=48 - / 7.6, 8.2 / 8.3   N=3200 K=1024 M=52 - / 7.2, 7.4 / 8.0
  //   N=4096 K=2048 M=25 6.9 / 7.2, 7.9 / 7.9   N=9600 K=1024 M=32 6.6 / 6.7, 7.4 / 7.8
  //   N=14336 K=512 M=25 6.6 / 5.5, 6.8 / 6.4, M=40 6.5 / 6.3, 6.7 / 7.1, M=64 6.5 / 7.2, 6.8 / 8.0
  const int64_t ctas = tiles * split;
  const bool captured = use == SmallUse::kLinearInGraph || use == SmallUse::kCodesInGraph;
  if (M <= 16) {
    if (M * own > 256) return s;
  } else if (ctas <= 64) {
    if (M * own > 128 || (stages <= 4 && M > (captured ? 44 : 60))) return s;
  } else if (split == 1) {
    if (M * own > (captured ? 96 : 112) || M > (captured ? 32 : 48)) return s;
  } else if (M * own > 112 || M > (ctas > 110 ? 24 : captured && stages <= 4 ? 44 : 56)) {
    return s;
  }
  // On codes that are there already no launch is saved.  In a graph the longer way to the first MMA is not hidden behind the kernel before, so
  // that only long K pays.  GEMM, us eager and from a graph (general kernel / so): M=8 N=512 K=1024 4.1 / 3.6, 4.6 / 5.2; M=24 N=512 K=1536
  // 4.7 / 4.2, 5.2 / 5.8; M=8 N=4096 K=1024 4.1 / 4.8, 4.7 / 5.4; M=32 N=2048 K=512 3.5 / 4.4, 4.1 / 5.7; M=8 N=14336 K=4096 12.2 / 9.5, 12.0 / 10.6;
  // M=16 of that 12.0 / 10.0, 12.3 / 11.2.
  const bool linear = use == SmallUse::kLinear || use == SmallUse::kLinearInGraph;
  const bool pays = linear         ? true
                    : captured     ? M <= (own >= 16 ? 16 : 8) && stages >= 8 && own >= 3
                    : stages < 4   ? M <= 4
                    : split == 1   ? M <= 8 || own >= 16
                    : ctas <= 64   ? M <= (stages < 6 ? 16 : 24)
                                   : M <= 8 && own >= 3;
  if (!pays) return s;
  int ring = own < kRingMost ? own : kRingMost;
  while (ring > 0 && small_layout(ring, own, m_pad, (int)M, split).bytes + 1024 > kSmemMost) --ring;
  if (ring < (own < 4 ? own : 4)) return s;
  s.split = split;
  s.ring = ring;
  s.stages = (int)stages;
  s.m_pad = m_pad;
  s.smem = small_layout(ring, own, m_pad, (int)M, split).bytes + 1024;
  s.ok = true;
  return s;
}

int launch_gemm_small(const SmallPlan& plan, const CUtensorMap& mw, const void* x, int x_dtype, int64_t ldx, const float* gs, const uint8_t* x_sf,
                      const uint8_t* w_sf, const float* alpha, void* out, int out_dtype, int M, int N, int K, int* status, cudaStream_t st) {
  SmallParams p = {};
  p.x = x;
  p.ldx = ldx;
  p.gs = gs;
  p.x_sf = x_sf;
  p.w_sf = w_sf;
  p.alpha = alpha;
  p.out = out;
  p.out_dtype = out_dtype;
  p.load32 = aligned(x, 32) && ldx % 16 == 0;
  p.M = M;
  p.N = N;
  p.K = K;
  p.m_pad = plan.m_pad;
  p.split = plan.split;
  p.stages = plan.stages;
  p.ring = plan.ring;
  // four blocks of 16 per thread and stage, or fewer where a CTA has not a stage for every group of warps
  const int own = (plan.stages + plan.split - 1) / plan.split;
  int wps = M <= 8 ? 1 : (M <= 16 ? 2 : (M <= 32 ? 4 : 8));
  while (wps * own < kXWarps && wps * 2 < M) wps *= 2;
  p.warps_per_stage = wps;
  uint32_t cols = 32;
  while (cols < (uint32_t)((plan.m_pad + 31) & ~31) + 32u * plan.ring) cols *= 2;
  p.tmem_cols = cols;
  p.status = status;
  const unsigned grid = (unsigned)((N + 127) / 128 * plan.split);
  if (gs == nullptr) return launch_small_t<__half, true>(mw, p, grid, plan.smem, st);
  return x_dtype == B200FP4_DTYPE_BF16 ? launch_small_t<__nv_bfloat16, false>(mw, p, grid, plan.smem, st)
                                       : launch_small_t<__half, false>(mw, p, grid, plan.smem, st);
}

}  // namespace b200fp4
