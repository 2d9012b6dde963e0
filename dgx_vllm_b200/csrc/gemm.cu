// Dense block-scaled NVFP4 GEMM for sm_100a: out[M,N] = alpha * (A . sfA)(B . sfB)^T
//
// Replaces the GEMM behind cuda_fp4_gemm.h / cutlass_scaled_fp4_mm in the reference (whose own
// kernels are scalar CUDA-core loops, cutlass_nvfp4/nvfp4_gemm_kernel.cuh:296-345) with a
// tcgen05 design:
//   * persistent, warp-specialised CTAs (one per SM): three warps issue the copies, one issues
//     tcgen05.mma, further warps, in groups of four, move scale factors and run the epilogue;
//   * operands are packed E2M1 bytes, K-major, staged by 2-D TMA (no multicast) into 128-byte
//     swizzled shared-memory tiles of 128 (A) / BN (B) rows x 256 k; scale factors come from the
//     128x4-tile swizzled global layout, where the 4 k-blocks x 128 rows an MMA needs are 512
//     contiguous bytes: one bulk copy per stage brings them to shared memory and four dedicated
//     warps (one per 32-lane quarter of tensor memory) move them on with tcgen05.st, which keeps
//     them off the tensor pipe (a tcgen05.cp per scale tile measured ~36 cycles there, a quarter
//     of an MMA);
//   * tcgen05.mma.kind::mxf4nvf4.block_scale (M=128, N=BN, K=64) accumulates fp32 in tensor
//     memory; the epilogue reads it with tcgen05.ld, multiplies by alpha and writes bf16/f16;
//   * BN=128 double-buffers the accumulator (epilogue of tile i overlaps the main loop of tile
//     i+1); BN=256 keeps one accumulator but drains it into packed registers and releases it before
//     the global stores, so only the ~1200-cycle drain is exposed; it moves 25 % fewer bytes per flop.
// Every mbarrier wait is bounded: on expiry the kernel records an error code in the status word
// and all roles drain out, so a protocol error cannot hang the GPU.
#include <cstring>
#include <mutex>
#include <type_traits>

#include "gemm_small.cuh"
#include "grouped.cuh"
#include "sm100_ptx.cuh"

namespace b200fp4 {

// CTA-pair (cta_group::2) kernel, gemm_pair.cu
int launch_gemm_pair(const CUtensorMap& ma, const CUtensorMap& mb, const uint8_t* sfa, const uint8_t* sfb, const float* alpha,
                     void* out, int out_bf16, int M, int N, int K, int* status, cudaStream_t st);

namespace {

constexpr int kBM = 128;
static_assert(kBM == kGroupTileRows, "tile list");
// Warp 0 copies of the operands, warp 1 MMA, warps 6-9 scale factors into tensor memory, the others epilogue in groups of four (one warp per 32-lane quarter of
// tensor memory): warps 2-5 and 10-13, and in the grouped kernels also 14-17 and 18-21.
constexpr int gemm_epi_groups(bool grouped) { return grouped ? 4 : 2; }
// The last warp issues the copies of scale factors (one thread issues a copy every 70-80 cycles and spends about 300 more per
// stage on its barriers).
constexpr int gemm_warps(bool grouped) { return 7 + 4 * gemm_epi_groups(grouped); }
constexpr int gemm_threads(bool grouped) { return 32 * gemm_warps(grouped); }
constexpr uint32_t kTmemCols = 512;

struct GemmParams {
  const uint8_t* sfa;   // swizzled [ceil(M/128)*128, ceil(K/64)*4]
  const uint8_t* sfb;   // swizzled [ceil(N/128)*128, ceil(K/64)*4]
  const float* alpha;
  void* out;
  int out_bf16;
  int out_f32;          // dense mode only: out is fp32 [M, N] (the accumulator times alpha, unrounded)
  int out_tma;          // dense 16-bit output through map_out: the epilogue stages tiles in shared memory and the copy
                        // engine writes whole lines (256-wide tiles only)
  int M, N, K;
  int m_tiles, n_tiles, k_stages;
  int* status;          // 0 = ok; otherwise the code of the wait that expired
  int early_b;          // dense mode: the kernel before this one writes neither B nor its scales
  // grouped (per-expert) mode: rows of A/out are permuted by expert, B is [E, N, K/2]
  const int* g_hdr;       // [0] = number of 128-row tiles over all experts
  const int4* g_mtiles;   // per 128-row tile: {first row, end row of its expert, scale-tile row of A, expert}
  const float* g_alphas;  // [E]
  long long g_sfb_expert_bytes;
  // fused SiLU(gate)*up + NVFP4 quantization of the result (grouped gate_up projection, N = 2*q_inter):
  // `out` receives packed codes [rows, q_inter/2], q_sf the swizzled block scales, q_gs[E] the global scales
  int q_inter;
  uint8_t* q_sf;
  const float* q_gs;
};

// What the roles need to know about one output tile.
struct TileInfo {
  int a_row0;       // first row of A / out
  int row_end;      // rows >= row_end are not stored
  int sfa_tile;     // index of the 128-row scale tile of A
  int b_row0;       // first row of the (flattened) B matrix
  int sfb_tile0;    // index of the first 128-row scale tile of B inside its expert
  int sfb_tile1;    // ... of the second one (256-wide tiles)
  int b_row1;       // fused SiLU tiles: first row of the "up" half of B (the gate half starts at b_row0)
  int expert;       // -1 in dense mode
  int n0;           // first output column
};

template <int BN, bool kGrouped, bool kSiluQuant = false>
__device__ __forceinline__ TileInfo tile_info(const GemmParams& p, int tile, int m_tiles) {
  TileInfo t;
  // Dense: row tiles fastest, so that the CTAs of a round share few column tiles of B.  Grouped: column tiles fastest -- the
  // rows of a tile and the weights of its expert are then both read from HBM once (with row tiles fastest the permuted
  // activations came back from HBM for every column tile: 1004 MB read instead of about 700 for the gate_up projection of
  // 81,920 rows, 2048 x 1024, 512 experts).
  const int mt = kGrouped ? tile / p.n_tiles : tile % m_tiles, nt = kGrouped ? tile - mt * p.n_tiles : tile / m_tiles;
  if (kSiluQuant) {
    // tile nt pairs gate columns [128 nt, +128) with up columns q_inter + [128 nt, +128); n0 counts output columns
    const int4 r = p.g_mtiles[mt];
    t.n0 = nt * 128;
    t.sfb_tile0 = nt;
    t.sfb_tile1 = p.q_inter / 128 + nt;
    t.a_row0 = r.x;
    t.row_end = r.y;
    t.sfa_tile = r.z;
    t.expert = r.w;
    t.b_row0 = r.w * p.N + nt * 128;
    t.b_row1 = t.b_row0 + p.q_inter;
    return t;
  }
  t.n0 = nt * BN;
  t.sfb_tile0 = nt * (BN / 128);
  t.sfb_tile1 = t.sfb_tile0 + 1;
  t.b_row1 = 0;
  if (kGrouped) {
    const int4 r = p.g_mtiles[mt];
    t.a_row0 = r.x;
    t.row_end = r.y;
    t.sfa_tile = r.z;
    t.expert = r.w;
    t.b_row0 = r.w * p.N + nt * BN;
  } else {
    t.a_row0 = mt * kBM;
    t.row_end = p.M;
    t.sfa_tile = mt;
    t.expert = -1;
    t.b_row0 = nt * BN;
  }
  return t;
}

// 16 NB gate and as many up values of one row (as 16-bit pairs) -> SiLU(gate)*up rounded to T -> NB NVFP4 blocks:
// 2 NB words of codes and NB scale bytes, with the arithmetic of the stand-alone SiLU-mul quantizer.
template <typename T, int NB>
__device__ __forceinline__ void silu_quant_row(const uint32_t* pg, const uint32_t* pu, float gs, float rcp_gs,
                                               uint32_t* codes, uint32_t& sf4) {
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    float x[16];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t wg = pg[b * 8 + i], wu = pu[b * 8 + i];
      float g0, g1, u0, u1;
      if (sizeof(T) == 2 && std::is_same<T, __nv_bfloat16>::value) {
        g0 = __uint_as_float(wg << 16); g1 = __uint_as_float(wg & 0xFFFF0000u);
        u0 = __uint_as_float(wu << 16); u1 = __uint_as_float(wu & 0xFFFF0000u);
      } else {
        const float2 fg = __half22float2(*reinterpret_cast<const __half2*>(&wg));
        const float2 fu = __half22float2(*reinterpret_cast<const __half2*>(&wu));
        g0 = fg.x; g1 = fg.y; u0 = fu.x; u1 = fu.y;
      }
      x[2 * i] = to_f32<T>(from_f32<T>(silu_f32(g0) * u0));
      x[2 * i + 1] = to_f32<T>(from_f32<T>(silu_f32(g1) * u1));
    }
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(x[i]));
    float scale = __fmul_rn(gs, __fmul_rn(amax, 0.16666667163372039794921875f));
    scale = fminf(scale, 448.f);
    const uint8_t sfb = f32_to_e4m3(scale);
    const float os = out_scale_of(sfb, rcp_gs);
    codes[b * 2] = f32x8_to_e2m1(__fmul_rn(x[0], os), __fmul_rn(x[1], os), __fmul_rn(x[2], os), __fmul_rn(x[3], os),
                                 __fmul_rn(x[4], os), __fmul_rn(x[5], os), __fmul_rn(x[6], os), __fmul_rn(x[7], os));
    codes[b * 2 + 1] = f32x8_to_e2m1(__fmul_rn(x[8], os), __fmul_rn(x[9], os), __fmul_rn(x[10], os), __fmul_rn(x[11], os),
                                     __fmul_rn(x[12], os), __fmul_rn(x[13], os), __fmul_rn(x[14], os), __fmul_rn(x[15], os));
    sf4 |= (uint32_t)sfb << (8 * b);
  }
}

// 32 finished columns of one row of the dense output
__device__ __forceinline__ void store_row32(const GemmParams& p, int row, int col0, const float (&v)[32]) {
  if (col0 >= p.N) return;
  const bool whole = col0 + 32 <= p.N;
  if (p.out_f32) {
    float* dst = reinterpret_cast<float*>(p.out) + (size_t)row * p.N + col0;
    if (whole && (p.N % 4) == 0) {
#pragma unroll
      for (int i = 0; i < 8; ++i) reinterpret_cast<float4*>(dst)[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (col0 + i < p.N) dst[i] = v[i];
    }
    return;
  }
  uint32_t w[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    if (p.out_bf16) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&h);
    } else {
      const __half2 h = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
  }
  uint16_t* dst = reinterpret_cast<uint16_t*>(p.out) + (size_t)row * p.N + col0;
  if (whole && (p.N % 8) == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) reinterpret_cast<uint4*>(dst)[i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (col0 + i < p.N) dst[i] = (uint16_t)((i & 1) ? (w[i >> 1] >> 16) : (w[i >> 1] & 0xFFFFu));
  }
}

// ---------------------------------------------------------------------------------------- kernel

// BN = tile width; KB = 64-wide k-blocks (MMAs) per shared-memory stage.  Smaller stages do not change
// the bytes resident in shared memory but refill in finer steps, which keeps more of them in flight.
// kOutStage: bytes of shared memory the epilogue stages its output in.
template <int BN, int KB, int kOutStage = 0>
struct Cfg {
  static constexpr int kAcc = BN == 128 ? 2 : 1;                    // accumulator buffers in tensor memory
  static constexpr int kSfTiles = BN / 128;                         // 128-row scale tiles on the B side
  static constexpr int kRowBytes = KB * 32;                         // packed codes per row per stage
  static constexpr int kStageA = kBM * kRowBytes;
  static constexpr int kStageB = BN * kRowBytes;
  static constexpr int kStageSFA = KB * 512;
  static constexpr int kStageSFB = kSfTiles * KB * 512;
  static constexpr int kStageBytes = kStageA + kStageB + kStageSFA + kStageSFB;
  // as many stages as fit beside what the epilogue stages
  static constexpr int kFit = (227 * 1024 - 2048 - kOutStage) / kStageBytes, kMost = (BN == 128 ? 24 : 16) / KB;
  static constexpr int kStages = kFit < kMost ? kFit : kMost;
  // tensor-memory column map: accumulators, then one scale-factor block per shared-memory stage
  // (4 columns per k-block for A, 4*kSfTiles for B)
  static constexpr uint32_t kSfCols = KB * (4 + 4 * kSfTiles);
  static constexpr uint32_t kSfBase = kAcc * BN;
  static_assert(kSfBase + kStages * kSfCols <= 512, "tensor memory budget");
  static constexpr int kBarBytes = 1024;
  static constexpr size_t kSmemBytes = (size_t)kStages * kStageBytes + (size_t)kOutStage + 1024 /*alignment slack*/ + kBarBytes;
  // instruction descriptor: E2M1 x E2M1, UE4M3 scales, K-major A and B, N = BN, M = 128, dense K = 64
  static constexpr uint32_t kIdesc = (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
};

// Staging: the dense wide-tile kernel hands [32 rows x 64 columns] boxes of 8 warps to the copy engine.
// kSplit > 1: partial sums from the other CTAs of the cluster, 128 rows x 128 / kSplit columns fp32 each.
template <int BN, bool kGrouped, bool kSiluQuant, int kSplit = 1>
constexpr int out_stage_bytes() {
  return kSplit > 1 ? (kSplit - 1) * (4 / kSplit) * 16384 : (BN == 256 && !kGrouped ? 8 * 4096 : 0);
}

// One step of a transpose across lanes: a lane with its bit clear gives b for its partner's a, one with the bit set a for b
__device__ __forceinline__ void transpose4(uint32_t* a, uint32_t* b, bool bit, int mask) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t got = __shfl_xor_sync(0xffffffffu, bit ? a[i] : b[i], mask);
    if (bit) a[i] = got;
    else b[i] = got;
  }
}

// The KB scale tiles of a stage to tensor memory, `step` columns apart: all loads before the first store (one after the other
// they were on the path of short main loops: grouped down projection of 64 x 1280 rows, K = 1024, 96 us, 85 so)
template <int KB>
__device__ __forceinline__ void copy_sf(uint32_t tmem, uint32_t step, const unsigned char* sf, int lane) {
  uint4 w[KB];
#pragma unroll
  for (int kb = 0; kb < KB; ++kb) w[kb] = *reinterpret_cast<const uint4*>(sf + kb * 512 + lane * 16);
#pragma unroll
  for (int kb = 0; kb < KB; ++kb) tcgen05_st_32x32_x4(tmem + kb * step, w[kb]);
}

// kSplit > 1 (dense, 128-wide tiles, fewer tiles than SMs): the kSplit CTAs of a cluster each take a part of K of one tile; each
// then finishes 128 / kSplit of its columns, with the other CTAs' sums of them arriving through distributed shared memory.
// kStageSf: the scales of A come as [128-row tile][256 of k][row][16 bytes]
template <int BN, int KB, bool kGrouped, bool kSiluQuant = false, int kSplit = 1, bool kStageSf = false>
__global__ void __launch_bounds__(gemm_threads(kGrouped), 1)
    nvfp4_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                      const __grid_constant__ CUtensorMap map_out, const GemmParams p) {
  constexpr bool kOutTma = BN == 256 && !kGrouped && !kSiluQuant;     // the dense wide-tile kernel stores tiles through the copy engine
  constexpr int kOutStage = out_stage_bytes<BN, kGrouped, kSiluQuant, kSplit>();
  static_assert(kSplit == 1 || (BN == 128 && !kGrouped && (kSplit == 2 || kSplit == 4)), "split K");
  using C = Cfg<BN, KB, kOutStage>;
  constexpr int kEpi = gemm_epi_groups(kGrouped);
  extern __shared__ unsigned char smem_raw[];
  // 1024-byte alignment for the 128-byte swizzle atoms
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* out_stage = smem + (size_t)C::kStages * C::kStageBytes;      // 1024-byte aligned (stages are multiples of 1 KiB)
  uint64_t* bars = reinterpret_cast<uint64_t*>(out_stage + kOutStage);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + C::kStages;
  uint64_t* acc_full = bars + 2 * C::kStages;
  uint64_t* acc_empty = acc_full + C::kAcc;
  uint64_t* sf_full = acc_empty + C::kAcc;     // scale factors of the stage have landed (before the operands)
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(sf_full + C::kStages);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 5);       // the operand copies, and each scale-factor warp
      mbar_init(smem_u32(&empty_bar[s]), 1);
      mbar_init(smem_u32(&sf_full[s]), 1);
    }
    for (int a = 0; a < C::kAcc; ++a) {
      mbar_init(smem_u32(&acc_full[a]), 1);
      mbar_init(smem_u32(&acc_empty[a]), 4 * kEpi);      // one arrival per epilogue warp
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_ptr_smem)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  if constexpr (kSplit > 1) cluster_sync_any();      // the other CTAs run before anything is sent to them
  else __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;
  constexpr int kWarpSf = gemm_warps(kGrouped) - 1;
  const int KT = (p.K + 63) / 64;   // 64-wide k-blocks = 512-byte scale tiles per 128 rows
  const int rank = kSplit > 1 ? (int)(blockIdx.x % kSplit) : 0;      // in the cluster
  const int first_tile = blockIdx.x / kSplit, tile_stride = gridDim.x / kSplit;
  const int ks_begin = p.k_stages * rank / kSplit, ks_end = p.k_stages * (rank + 1) / kSplit;
  // The weights of a linear layer do not depend on the quantizer that runs just before: the first ring of B and its scales is
  // requested while that kernel still runs (N=14336, K=4096: M=32 13.4 -> 12.1 us, M=128 13.4 -> 12.7).
  int early = 0;
  if (!kGrouped && p.early_b && (warp == 0 || warp == kWarpSf) && first_tile < p.m_tiles * p.n_tiles) {
    const bool elected = elect_one();
    const TileInfo ti = tile_info<BN, kGrouped, kSiluQuant>(p, first_tile, p.m_tiles);
    const uint8_t* sfb0 = p.sfb + (size_t)ti.sfb_tile0 * KT * 512;
    const uint8_t* sfb1 = p.sfb + (size_t)ti.sfb_tile1 * KT * 512;
    const int sf_tiles = C::kSfTiles == 1 || ti.sfb_tile1 * 128 >= p.N ? 1 : 2;
    early = min((int)C::kStages, ks_end - ks_begin);
    for (int s = 0; s < early; ++s) {
      const int ks = ks_begin + s;
      const uint32_t st = smem_u32(smem) + s * C::kStageBytes, sbar = smem_u32(&sf_full[s]), bar = smem_u32(&full_bar[s]);
      if (!elected) continue;
      if (warp == 0) {
        mbar_expect_tx(bar, (uint32_t)(C::kStageA + C::kStageB));
        tma_load_2d(st + C::kStageA, &map_b, ks * C::kRowBytes, ti.b_row0, bar);
      } else {
        const uint32_t bytes = (uint32_t)min(KB, KT - ks * KB) * 512, off = (uint32_t)ks * (KB * 512), dst = st + C::kStageA + C::kStageB;
        mbar_expect_tx(sbar, bytes * (1 + sf_tiles));
        bulk_load_1d(dst + C::kStageSFA, sfb0 + off, bytes, sbar);
        if (sf_tiles > 1) bulk_load_1d(dst + C::kStageSFA + KB * 512, sfb1 + off, bytes, sbar);
      }
    }
    __syncwarp();
  }
  pdl_wait();                 // everything above overlaps the end of the kernel before this one
  pdl_launch_dependents();
  // dense mode: the status word is cleared here instead of by a separate memset (a wait only writes it after its ~1 s
  // budget, long after this store); in grouped mode whoever made the tile list has cleared it
  if (!kGrouped && blockIdx.x == 0 && threadIdx.x == 0) *p.status = 0;
  const int m_tiles = kGrouped ? p.g_hdr[0] : p.m_tiles;
  const int n_tiles_total = m_tiles * p.n_tiles;
  float keep[kSplit > 1 ? 128 / kSplit : 1];                          // this thread's row of the columns its CTA finishes

  if (warp == 0 || warp == kWarpSf) {
    // ------------------------------------------------------------------ copies into shared memory: operands, scale factors
    const bool elected = elect_one();
    uint32_t s = 0, ph = 0;
    bool ok = true;
    for (int tile = first_tile; ok && tile < n_tiles_total; tile += tile_stride) {
      const TileInfo ti = tile_info<BN, kGrouped, kSiluQuant>(p, tile, m_tiles);
      const uint8_t* sfa = p.sfa + (size_t)ti.sfa_tile * (kStageSf ? p.k_stages * KB : KT) * 512;
      const uint8_t* sfb = p.sfb + (kGrouped ? (size_t)ti.expert * (size_t)p.g_sfb_expert_bytes : (size_t)0);
      const uint8_t* sfb0 = sfb + (size_t)ti.sfb_tile0 * KT * 512;
      const uint8_t* sfb1 = sfb + (size_t)ti.sfb_tile1 * KT * 512;
      const int sf_tiles = C::kSfTiles == 1 || ti.sfb_tile1 * 128 >= p.N ? 1 : 2;      // the second 128 columns may lie past N
      for (int ks = ks_begin; ks < ks_end; ++ks) {
        ok = mbar_wait_warp(smem_u32(&empty_bar[s]), ph ^ 1, p.status, 1);
        if (!ok) break;
        const bool b_requested = !kGrouped && early > 0;
        if (!kGrouped) --early;
        if (elected) {
          const uint32_t st = smem_u32(smem) + s * C::kStageBytes, bar = smem_u32(&full_bar[s]);
          if (warp == 0) {
            if (!b_requested) mbar_expect_tx(bar, (uint32_t)(C::kStageA + C::kStageB));
            tma_load_2d(st, &map_a, ks * C::kRowBytes, ti.a_row0, bar);
            if (!b_requested) tma_load_2d(st + C::kStageA, &map_b, ks * C::kRowBytes, ti.b_row0, bar);
            // with SiLU map_b's box is 128 rows: the gate rows and the up rows of the tile land one after the other
            if (kSiluQuant) tma_load_2d(st + C::kStageA + 128 * C::kRowBytes, &map_b, ks * C::kRowBytes, ti.b_row1, bar);
          } else {
            // scale factors have their own barrier, so that the scale warps can move them into tensor memory while the
            // operand tiles are still in flight
            const uint32_t bytes = (uint32_t)min(KB, KT - ks * KB) * 512, off = (uint32_t)ks * (KB * 512);
            const uint32_t bytes_a = kStageSf ? KB * 512 : bytes;
            const uint32_t sbar = smem_u32(&sf_full[s]), dst = st + C::kStageA + C::kStageB;
            if (!b_requested) mbar_expect_tx(sbar, bytes_a + bytes * sf_tiles);
            bulk_load_1d(dst, sfa + off, bytes_a, sbar);
            if (!b_requested) {
              bulk_load_1d(dst + C::kStageSFA, sfb0 + off, bytes, sbar);
              if (sf_tiles > 1) bulk_load_1d(dst + C::kStageSFA + KB * 512, sfb1 + off, bytes, sbar);
            }
          }
        }
        __syncwarp();
        if (++s == C::kStages) {
          s = 0;
          ph ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    // The warp can run only one or two MMAs ahead of the tensor core, so whatever it does between stages leaves the tensor
    // core idle: one barrier per stage (operands landed and scales in tensor memory), descriptors by addition, and the whole warp in
    // the loop (elect_one).
    const bool elected = elect_one();
    const uint64_t a_desc0 = desc_kmajor<C::kRowBytes>(smem_u32(smem)), b_desc0 = desc_kmajor<C::kRowBytes>(smem_u32(smem) + C::kStageA);
    const uint32_t full0 = smem_u32(full_bar);
    uint32_t s = 0, ph = 0, tcount = 0;
    bool ok = true;
    for (int tile = first_tile; ok && tile < n_tiles_total; tile += tile_stride, ++tcount) {
      const uint32_t acc = tcount % C::kAcc, aph = (tcount / C::kAcc) & 1;
      ok = mbar_wait_warp(smem_u32(&acc_empty[acc]), aph ^ 1, p.status, 2);
      if (!ok) break;
      const uint32_t d_tmem = tmem_base + acc * BN;
      for (int ks = ks_begin; ks < ks_end; ++ks) {
        ok = mbar_wait_warp(full0 + s * 8, ph, p.status, 3);
        if (!ok) break;
        tcgen05_fence_after();
        if (elected) {
          // each 64-wide k-block is 32 bytes further along the swizzled 128-byte rows (descriptors count 16 bytes)
          const uint64_t a_desc = a_desc0 + s * (C::kStageBytes >> 4), b_desc = b_desc0 + s * (C::kStageBytes >> 4);
          const uint32_t sfa_tmem = tmem_base + C::kSfBase + s * C::kSfCols, sfb_tmem = sfa_tmem + 4 * KB;
          const int kblocks = KT - ks * KB;
#pragma unroll
          for (int kb = 0; kb < KB; ++kb)
            if (kb < kblocks)
              tcgen05_mma_nvf4(d_tmem, a_desc + kb * 2, b_desc + kb * 2, C::kIdesc, sfa_tmem + kb * 4, sfb_tmem + kb * (4 * C::kSfTiles),
                               (ks > ks_begin || kb > 0) ? 1u : 0u);
          tcgen05_commit(smem_u32(&empty_bar[s]));    // frees the stage when these MMAs have read it
          if (ks == ks_end - 1) tcgen05_commit(smem_u32(&acc_full[acc]));
        }
        __syncwarp();
        if (++s == C::kStages) {
          s = 0;
          ph ^= 1;
        }
      }
    }
  } else if (warp >= 6 && warp < 10) {
    // ------------------------------------------------------------------ scale factors (warps 6..9)
    // Each warp owns one 32-lane quarter of tensor memory.  Lane L needs row L of every 32x16-byte
    // scale tile (the four quarters hold identical copies), so each lane moves 16 bytes from shared
    // memory to its own lane with tcgen05.st -- this keeps the scale traffic off the tensor pipe,
    // where a tcgen05.cp per tile costs about a quarter of an MMA.
    const int quarter = warp & 3;
    uint32_t it = 0;
    bool ok = true;
    for (int tile = first_tile; ok && tile < n_tiles_total; tile += tile_stride) {
      for (int ks = ks_begin; ks < ks_end; ++ks, ++it) {
        const uint32_t s = it % C::kStages, ph = (it / C::kStages) & 1;
        ok = mbar_wait(smem_u32(&sf_full[s]), ph, p.status, 6);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tcgen05_fence_after();                     // the copy waited for the commit of the MMAs that read this slot's columns, and so has this
        const unsigned char* sf = smem + (size_t)s * C::kStageBytes + C::kStageA + C::kStageB;
        const uint32_t t0 = tmem_base + ((uint32_t)(quarter * 32) << 16) + C::kSfBase + s * C::kSfCols;
        const int kblocks = min(KB, KT - ks * KB);
        if (kblocks == KB) {
          if constexpr (kStageSf) {
            // 16 bytes of each of the rows lane, lane + 32, ...: a word per k-block
            static_assert(KB == 4, "stage of 256 k");
            uint4 w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = *reinterpret_cast<const uint4*>(sf + j * 512 + lane * 16);
            tcgen05_st_32x32_x4(t0, make_uint4(w[0].x, w[1].x, w[2].x, w[3].x));
            tcgen05_st_32x32_x4(t0 + 4, make_uint4(w[0].y, w[1].y, w[2].y, w[3].y));
            tcgen05_st_32x32_x4(t0 + 8, make_uint4(w[0].z, w[1].z, w[2].z, w[3].z));
            tcgen05_st_32x32_x4(t0 + 12, make_uint4(w[0].w, w[1].w, w[2].w, w[3].w));
          } else {
            copy_sf<KB>(t0, 4, sf, lane);
          }
#pragma unroll
          for (int j = 0; j < C::kSfTiles; ++j) copy_sf<KB>(t0 + 4 * KB + j * 4, 4 * C::kSfTiles, sf + C::kStageSFA + j * (KB * 512), lane);
        } else {
          for (int kb = 0; kb < kblocks; ++kb) {
            uint4 a;
            if constexpr (kStageSf) {
              const uint32_t* w = reinterpret_cast<const uint32_t*>(sf) + lane * 4 + kb;
              a = make_uint4(w[0], w[128], w[256], w[384]);
            } else {
              a = *reinterpret_cast<const uint4*>(sf + kb * 512 + lane * 16);
            }
            tcgen05_st_32x32_x4(t0 + kb * 4, a);
#pragma unroll
            for (int j = 0; j < C::kSfTiles; ++j)
              tcgen05_st_32x32_x4(t0 + 4 * KB + kb * (4 * C::kSfTiles) + j * 4,
                                  *reinterpret_cast<const uint4*>(sf + C::kStageSFA + j * (KB * 512) + kb * 512 + lane * 16));
          }
        }
        tcgen05_wait_st();
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&full_bar[s]));
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    // kEpi warps per tensor-memory lane quarter, each draining and storing its share of the tile's columns.
    // With long K the epilogue hides behind the next tile either way; with short K (the grouped down
    // projection: 8 MMAs per tile) the kernel is bound by how fast a tile can be drained and stored, and with SiLU and
    // quantization by the epilogue's arithmetic: about 3000 instructions per row and 64 columns keep eight warps busy for
    // longer than the tile's stages take (gate_up of 81,920 rows: 182 us with eight epilogue warps).
    const int quarter = warp & 3;                 // tensor-memory lanes [32*quarter, +32) belong to this warp
    constexpr int CH = BN / 32 / kEpi;            // 32-column chunks per warp
    const int grp = warp < 6 ? 0 : (warp - 6) >> 2;
    const int c_first = grp * CH;
    const float alpha_dense = kGrouped ? 0.f : p.alpha[0];
    uint32_t tcount = 0;
    bool ok = true;
    for (int tile = first_tile; ok && tile < n_tiles_total; tile += tile_stride, ++tcount) {
      const TileInfo ti = tile_info<BN, kGrouped, kSiluQuant>(p, tile, m_tiles);
      const float alpha = kGrouped ? p.g_alphas[ti.expert] : alpha_dense;
      const uint32_t acc = tcount % C::kAcc, aph = (tcount / C::kAcc) & 1;
      ok = mbar_wait(smem_u32(&acc_full[acc]), aph, p.status, 4);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tcgen05_fence_after();
      const int row = ti.a_row0 + quarter * 32 + lane;
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * BN;
      if constexpr (kSiluQuant) {
        // Tensor-memory columns [0,128) hold the gate half of this thread's row, [128,256) the up half.
        // This warp takes 32 of the 128 output columns: 2 blocks of 16 -> 16 bytes of codes + 2 scale bytes,
        // computed exactly as the separate SiLU-mul quantizer does from the 16-bit rounded GEMM output.
        const float gs = p.q_gs[ti.expert];
        const float rcp_gs = __frcp_rn(gs + (gs == 0.f ? 1.0e8f : 0.f));
        // read both halves, hand the accumulator back, and only then round to 16-bit pairs (as the separate GEMM's output is)
        // and do the SiLU / quantization arithmetic, so that all of it overlaps the next tile's main loop
        uint32_t rg[32], ru[32];
        tcgen05_ld_32x32(taddr + grp * 32, rg);
        tcgen05_ld_32x32(taddr + 128 + grp * 32, ru);
        tcgen05_wait_ld();
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&acc_empty[acc]));
        uint32_t pg[16], pu[16];
        pack_row(rg, alpha, p.out_bf16 != 0, pg);
        pack_row(ru, alpha, p.out_bf16 != 0, pu);
        // rows past the end of the expert are never stored: warps whose 32 rows are all past it skip the arithmetic
        if (row < ti.row_end) {
          uint32_t codes[4];
          uint32_t sf2 = 0;
          if (p.out_bf16) silu_quant_row<__nv_bfloat16, 2>(pg, pu, gs, rcp_gs, codes, sf2);
          else silu_quant_row<__half, 2>(pg, pu, gs, rcp_gs, codes, sf2);
          const int col = ti.n0 + grp * 32;
          uint8_t* dst = reinterpret_cast<uint8_t*>(p.out) + (size_t)row * (size_t)(p.q_inter / 2) + col / 2;
          *reinterpret_cast<uint4*>(dst) = make_uint4(codes[0], codes[1], codes[2], codes[3]);
          const size_t kt2 = (size_t)(p.q_inter / 64);
          *reinterpret_cast<uint16_t*>(p.q_sf + ((size_t)ti.sfa_tile * kt2 + (size_t)(col / 64)) * 512 + lane * 16 + quarter * 4 +
                                       (grp & 1) * 2) = (uint16_t)sf2;
        }
        continue;
      }
      if constexpr (kSplit > 1) {
        // 32-column chunk c of the tile belongs to CTA c * kSplit / 4: kept if that is this one, sent there otherwise as
        // [sender][chunk][quarter][four columns][row]: a warp's store of four columns is 512 contiguous bytes (a column at a time, 128 bytes,
        // the exchange took four times as many stores to another SM)
        constexpr int kOwn = 4 / kSplit;
#pragma unroll
        for (int c = 0; c < CH; ++c) {
          const int chunk = c_first + c, owner = chunk / kOwn;
          uint32_t r[32];
          tcgen05_ld_32x32(taddr + chunk * 32, r);
          tcgen05_wait_ld();
          if (owner == rank) {
#pragma unroll
            for (int i = 0; i < 32; ++i) keep[(kOwn == 1 ? 0 : c * 32) + i] = __uint_as_float(r[i]);
          } else if (row < ti.row_end) {
            const int slot = rank < owner ? rank : rank - 1;
            const uint32_t dst = map_to_cta(smem_u32(out_stage) + (uint32_t)((slot * kOwn + chunk % kOwn) * 4 + quarter) * 4096u + lane * 16u,
                                            (uint32_t)owner);
#pragma unroll
            for (int i = 0; i < 8; ++i)
              asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + i * 512u), "r"(r[4 * i]), "r"(r[4 * i + 1]),
                           "r"(r[4 * i + 2]), "r"(r[4 * i + 3])
                           : "memory");
          }
        }
        continue;
      }
      if (!kGrouped && p.out_f32) {
        // fp32 output (the cudaFP4GemmEx form): each 32-column chunk goes straight from tensor memory to global
        // memory; the accumulator is handed back after the last chunk
        float* dst_row = reinterpret_cast<float*>(p.out) + (size_t)row * p.N;
#pragma unroll 1
        for (int c = 0; c < CH; ++c) {
          uint32_t r[32];
          tcgen05_ld_32x32(taddr + (c_first + c) * 32, r);
          tcgen05_wait_ld();
          const int col0 = ti.n0 + (c_first + c) * 32;
          if (row < ti.row_end && col0 < p.N) {
            if (col0 + 32 <= p.N && (p.N % 4) == 0) {
#pragma unroll
              for (int i = 0; i < 8; ++i)
                reinterpret_cast<float4*>(dst_row + col0)[i] =
                    make_float4(__uint_as_float(r[4 * i]) * alpha, __uint_as_float(r[4 * i + 1]) * alpha,
                                __uint_as_float(r[4 * i + 2]) * alpha, __uint_as_float(r[4 * i + 3]) * alpha);
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (col0 + i < p.N) dst_row[col0 + i] = __uint_as_float(r[i]) * alpha;
            }
          }
        }
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&acc_empty[acc]));
        continue;
      }
      // Drain this thread's row of the accumulator into packed 16-bit registers, two loads of 32 columns in flight; the
      // accumulator goes back to the MMA warp after the last loads, before their conversion and the stores, which then
      // overlap the next tile's main loop.
      uint32_t packed[16 * CH];
#pragma unroll
      for (int c = 0; c < CH; c += 2) {
        uint32_t r0[32], r1[32];
        tcgen05_ld_32x32(taddr + (c_first + c) * 32, r0);
        if (c + 1 < CH) tcgen05_ld_32x32(taddr + (c_first + c + 1) * 32, r1);
        tcgen05_wait_ld();
        if (c + 2 >= CH) {
          tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&acc_empty[acc]));
        }
        pack_row(r0, alpha, p.out_bf16 != 0, packed + c * 16);
        if (c + 1 < CH) pack_row(r1, alpha, p.out_bf16 != 0, packed + (c + 1) * 16);
      }
      if constexpr (kOutTma) if (p.out_tma) {
        // This warp's 32 rows x 128 columns leave in two halves of 64 columns (128 bytes per row): rows go to a private
        // staging buffer with the 128-byte swizzle of the tensor map (16-byte chunk c of row r at c ^ (r % 8): the
        // lanes of a warp write different banks), one lane hands the box to the copy engine, which writes whole lines
        // and clips rows / columns beyond the tensor.
        const uint32_t stg = smem_u32(out_stage) + (uint32_t)(grp * 4 + quarter) * 4096u;
        const int row0 = ti.a_row0 + quarter * 32;
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          if (lane == 0) bulk_wait_read0();          // the previous box has left the buffer
          __syncwarp();
#pragma unroll
          for (int c = 0; c < 8; ++c)
            sts128(stg + (uint32_t)lane * 128u + (uint32_t)((c ^ (lane & 7)) << 4), packed[hh * 32 + 4 * c],
                   packed[hh * 32 + 4 * c + 1], packed[hh * 32 + 4 * c + 2], packed[hh * 32 + 4 * c + 3]);
          fence_proxy_async_smem();
          __syncwarp();
          const int col0 = ti.n0 + (c_first * 32) + hh * 64;
          if (lane == 0 && col0 < p.N && row0 < p.M) {
            tma_store_2d(&map_out, col0, row0, stg);
            bulk_commit();
          }
        }
        continue;
      }
      if constexpr (kGrouped) if ((p.N % 8) == 0) {
        // Rows of the next expert must not be touched, so the copy engine's boxes do not fit; a lane that stored its own row
        // directly would write 32 rows per instruction, 32 bytes each.  Instead four neighbouring lanes turn their rows' 16-byte
        // chunks around by shuffles, and each stores its chunk of all four.  (Turned around in shared memory, the 32 KB of
        // buffers cost the fourth stage of the ring: 81,920 rows x 2048 x 512 138 us, 132 so; 8192 rows x 1024 x 1024, 64
        // experts, 81 us, 73 so.  The tile in two halves of 128 columns, one drained while the other is computed: 163.)
        const int row0 = ti.a_row0 + quarter * 32 + (lane & ~3);
#pragma unroll
        for (int c = 0; c < CH; ++c) {
          uint32_t* w = packed + c * 16;
          transpose4(w, w + 4, lane & 1, 1);
          transpose4(w + 8, w + 12, lane & 1, 1);
          transpose4(w, w + 8, lane & 2, 2);
          transpose4(w + 4, w + 12, lane & 2, 2);
          const int col = ti.n0 + (c_first + c) * 32 + (lane & 3) * 8;
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (row0 + i < ti.row_end && col < p.N)
              *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.out) + (size_t)(row0 + i) * p.N + col) =
                  make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
        }
        continue;
      }
      if (row < ti.row_end) {
        uint16_t* dst_row = reinterpret_cast<uint16_t*>(p.out) + (size_t)row * p.N;
#pragma unroll
        for (int c = 0; c < CH; ++c) {
          const int col0 = ti.n0 + (c_first + c) * 32;
          if (col0 < p.N) {
            uint16_t* dst = dst_row + col0;
            if (col0 + 32 <= p.N && (p.N % 16) == 0 && (reinterpret_cast<uintptr_t>(dst) & 31) == 0) {
              // 32-byte stores: whole sectors, half as many store instructions as 16-byte ones
#pragma unroll
              for (int i = 0; i < 2; ++i)
                st_global_v8(dst + 16 * i, &packed[c * 16 + 8 * i]);
            } else if (col0 + 32 <= p.N && (p.N % 8) == 0) {
#pragma unroll
              for (int i = 0; i < 4; ++i)
                reinterpret_cast<uint4*>(dst)[i] = make_uint4(packed[c * 16 + 4 * i], packed[c * 16 + 4 * i + 1],
                                                              packed[c * 16 + 4 * i + 2], packed[c * 16 + 4 * i + 3]);
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (col0 + i < p.N)
                  dst[i] = (uint16_t)((i & 1) ? (packed[c * 16 + (i >> 1)] >> 16) : (packed[c * 16 + (i >> 1)] & 0xFFFFu));
            }
          }
        }
      }
    }
  }
  if constexpr (kSplit > 1) {
    // every CTA's sums have arrived (also after a timed-out wait: the status word then says that the result is not valid)
    // Over two CTAs the sums and the two kept chunks take 128 registers and spill 40 bytes.  Four values at a time onto what is kept, 122 registers
    // and no spills, took 1 to 2 % longer (28 sizes: 256x4096x4096 7.77 / 7.95 us, 323x1536x7616 9.69 / 9.86).
    __syncwarp();
    cluster_sync_any();
    constexpr int kOwn = 4 / kSplit;
    const int quarter = warp & 3, grp = warp < 6 ? 0 : (warp - 6) >> 2;
    const bool epilogue = warp >= 2 && (warp < 6 || (warp >= 10 && warp < 14));
    if (epilogue && grp == rank * 2 / kSplit && first_tile < n_tiles_total) {
      const TileInfo ti = tile_info<BN, kGrouped, kSiluQuant>(p, first_tile, m_tiles);
      const int row = ti.a_row0 + quarter * 32 + lane;
      const float alpha = p.alpha[0];
      if (row < ti.row_end) {
#pragma unroll
        for (int c = 0; c < kOwn; ++c) {
          float v[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = 0.f;
#pragma unroll
          for (int src = 0; src < kSplit; ++src) {           // in the order of K
            if (src == rank) {
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] += keep[c * 32 + i];
            } else {
              const int slot = src < rank ? src : src - 1;
              const uint32_t at = smem_u32(out_stage) + (uint32_t)((slot * kOwn + c) * 4 + quarter) * 4096u + lane * 16u;
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const uint4 x = lds128(at + i * 512u);
                v[4 * i] += __uint_as_float(x.x);
                v[4 * i + 1] += __uint_as_float(x.y);
                v[4 * i + 2] += __uint_as_float(x.z);
                v[4 * i + 3] += __uint_as_float(x.w);
              }
            }
          }
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] *= alpha;
          store_row32(p, row, ti.n0 + (rank * kOwn + c) * 32, v);
        }
      }
    }
  }
  // all roles fall through to here (also after a timed-out wait), so tensor memory is always freed
  if (kOutTma && p.out_tma && lane == 0 && warp >= 2 && (warp < 6 || warp >= 10)) bulk_wait0();
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

// ---------------------------------------------------------------------------------------- grouped helpers


// One block: cuts every expert's row range into 128-row tiles.
//   hdr[0] = number of tiles; mtiles[t] = {first row, end row of the expert, A scale-tile row, expert}
__global__ void __launch_bounds__(1024)
    grouped_tiles_kernel(const int* __restrict__ expert_offsets, const int* __restrict__ sf_offsets, int E, int* hdr,
                         int4* mtiles, int max_tiles) {
  __shared__ int s_scan[1024];
  __shared__ int s_base;
  const int tid = threadIdx.x;
  if (tid == 0) s_base = 0;
  // the four ints in front of hdr are the GEMM's status word (0 = ok) and its padding: cleared here with hdr, so the
  // call needs no separate memset
  if (tid < 8) hdr[tid - 4] = 0;
  __syncthreads();
  for (int e0 = 0; e0 < E; e0 += 1024) {
    const int e = e0 + tid;
    int rows = 0, first = 0;
    if (e < E) {
      first = expert_offsets[e];
      rows = expert_offsets[e + 1] - first;
    }
    const int nt = (rows + kBM - 1) / kBM;
    s_scan[tid] = nt;
    __syncthreads();
    for (int d = 1; d < 1024; d <<= 1) {          // inclusive Hillis-Steele scan
      const int v = tid >= d ? s_scan[tid - d] : 0;
      __syncthreads();
      s_scan[tid] += v;
      __syncthreads();
    }
    const int start = s_base + s_scan[tid] - nt;
    if (e < E) {
      const int sf_row_tile = sf_offsets[e] / 128;
      for (int i = 0; i < nt; ++i)
        if (start + i < max_tiles) mtiles[start + i] = make_int4(first + i * kBM, first + rows, sf_row_tile + i, e);
    }
    __syncthreads();
    if (tid == 1023) s_base += s_scan[1023];
    __syncthreads();
  }
  if (tid == 0) hdr[0] = min(s_base, max_tiles);
}

// out[i, :] = in[dst2src[i] / src_div, :] for 16-byte chunks; rows whose map entry is < 0 become zero.
__global__ void shuffle_rows_kernel(const uint4* __restrict__ in, const int* __restrict__ dst2src, int src_div,
                                    int64_t chunks_per_row, int64_t n_dst, uint4* __restrict__ out) {
  const int64_t total = n_dst * chunks_per_row;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / chunks_per_row, c = i - r * chunks_per_row;
    const int src = dst2src[r];
    out[i] = src >= 0 ? in[(int64_t)(src / src_div) * chunks_per_row + c] : make_uint4(0, 0, 0, 0);
  }
}

// ---------------------------------------------------------------------------------------- host

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    fn = reinterpret_cast<EncodeTiledFn>(sym);
  }
  return fn;
}

// Encoded maps are remembered by their arguments (a weight is encoded once, not once per call).
struct MapKey {
  const void* base;
  uint64_t rows, row_bytes, row_stride;
  uint32_t box_rows;
  int box_bytes;
};
struct MapCache {
  static constexpr int kSlots = 64;
  MapKey key[kSlots];
  CUtensorMap map[kSlots];
  bool used[kSlots] = {false};
  std::mutex mu;
};
MapCache g_map_cache;

bool encode_rows_map(CUtensorMap* map, const MapKey& k) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {k.row_bytes, k.rows};
  cuuint64_t strides[1] = {k.row_stride};
  cuuint32_t box[2] = {(cuuint32_t)k.box_bytes, k.box_rows};
  const CUtensorMapSwizzle sw = k.box_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                                : (k.box_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
  cuuint32_t estr[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(k.base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool make_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t row_bytes, uint32_t box_rows, int box_bytes) {
  return make_rows_map(map, base, rows, row_bytes, row_bytes, box_rows, box_bytes);
}

// [rows, cols] 16-bit row-major output; box = 64 columns (128 bytes) x 32 rows, 128-byte swizzle
bool make_out_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {cols * 2};
  cuuint32_t box[2] = {64, 32};
  cuuint32_t estr[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

bool make_rows_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t row_bytes, uint64_t row_stride, uint32_t box_rows,
                   int box_bytes) {
  const MapKey k{base, rows, row_bytes, row_stride, box_rows, box_bytes};
  const size_t h = (reinterpret_cast<uintptr_t>(base) >> 8) * 0x9E3779B97F4A7C15ull + rows * 31 + box_rows;
  const int slot = (int)(h % MapCache::kSlots);
  std::lock_guard<std::mutex> lock(g_map_cache.mu);
  if (g_map_cache.used[slot] && memcmp(&g_map_cache.key[slot], &k, sizeof(MapKey)) == 0) {
    *map = g_map_cache.map[slot];
    return true;
  }
  if (!encode_rows_map(map, k)) return false;
  memset(&g_map_cache.key[slot], 0, sizeof(MapKey));
  g_map_cache.key[slot] = k;
  g_map_cache.map[slot] = *map;
  g_map_cache.used[slot] = true;
  return true;
}

namespace {

template <int BN, int KB, bool kGrouped, bool kSiluQuant = false, int kSplit = 1, bool kStageSf = false>
int launch_gemm(const CUtensorMap& ma, const CUtensorMap& mb, GemmParams p, int max_m_tiles, cudaStream_t st,
                const CUtensorMap* mo = nullptr) {
  using C = Cfg<BN, KB, out_stage_bytes<BN, kGrouped, kSiluQuant, kSplit>()>;
  CUtensorMap dummy = {};
  if (mo == nullptr) {
    mo = &dummy;
    p.out_tma = 0;
  }
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    if (cudaFuncSetAttribute(nvfp4_gemm_kernel<BN, KB, kGrouped, kSiluQuant, kSplit, kStageSf>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)C::kSmemBytes) != cudaSuccess) {
      cudaGetLastError();
      return B200FP4_STATUS_EXECUTION_FAILED;
    }
    attr_set[dev] = true;
  }
  p.n_tiles = kSiluQuant ? p.q_inter / 128 : (p.N + BN - 1) / BN;
  long long grid = (long long)max_m_tiles * p.n_tiles;
  if (kSplit == 1 && grid > sm_count()) grid = sm_count();
  if (grid < 1) grid = 1;
  p.k_stages = (p.K + KB * 64 - 1) / (KB * 64);
  if (launch_pdl_cluster(kSplit, nvfp4_gemm_kernel<BN, KB, kGrouped, kSiluQuant, kSplit, kStageSf>, dim3((unsigned)grid * kSplit),
                         dim3(gemm_threads(kGrouped)), C::kSmemBytes, st, ma, mb, *mo, p) != cudaSuccess) {
    cudaGetLastError();
    return B200FP4_STATUS_EXECUTION_FAILED;
  }
  return B200FP4_STATUS_SUCCESS;
}

// 64-wide k-blocks per shared-memory stage.  The kernel template also builds with 2 or 1 (64- and
// 32-byte swizzled rows, 8 or 16 stages); on B200 those measured 190 and 317 us against 150 us at
// M=4096 (TMA issues one request per box row, so narrower rows double and quadruple the requests).
constexpr int kStageKb = 4;

// Clusters of four CTAs of the kernel that splits K, which run at once
int resident_splits_of_four() {
  static ResidentClusters counts[64];
  return resident_clusters_of(counts, nvfp4_gemm_kernel<128, kStageKb, false, false, 4>, 4, gemm_threads(false),
                              (size_t)Cfg<128, kStageKb, out_stage_bytes<128, false, false, 4>()>::kSmemBytes);
}

// Tile of the dense GEMM: 128- or 256-wide on single CTAs (one per SM), 256 x 256 on CTA pairs, and for few tiles the split of K
// over clusters of two or four.  Each takes whole rounds over the SMs, so the choice is the least of
//   fixed + rounds x (stages x time per 256-k stage + tile)
// with times in us fitted to sweeps on B200 (weights cold, M 128..4096, N 2048..16000, K 512..8192; within 10 % of all but the
// ragged sizes).  What the former rule (256-wide once there are as many of them as SMs, pairs likewise) cost: M=777, N=3000,
// K=4160 168 narrow tiles on 148 SMs 20.7 us, 84 wide ones 13.4; M=1024, N=4096, K=4096 17.8 / 12.4; M=600, N=6000, K=8192
// 30.5 us, pairs 19.3.
void pick_dense_tile(int64_t M, int64_t N, int64_t stages, bool f32, int& bn, int& split) {
  const int64_t sms = sm_count(), m128 = (M + 127) / 128, m256 = (M + 255) / 256, n128 = (N + 127) / 128, n256 = (N + 255) / 256;
  auto rounds = [](int64_t tiles, int64_t places) { return (double)((tiles + places - 1) / places); };
  const double S = (double)stages;
  const double narrow = 3.3 + rounds(m128 * n128, sms) * (0.42 * S + 0.6);
  const double wide = 3.3 + rounds(m128 * n256, sms) * (0.56 * S + 0.6);
  // a row pitch that is no multiple of 32 bytes slows the pair kernel's direct stores
  const double pair = 3.8 + rounds(m256 * n256, sms / 2) * (0.46 * S + 1.6 + (N % 16 != 0 ? 1.5 : 0.0));
  bn = wide < narrow ? 256 : 128;
  if (!f32 && pair < (wide < narrow ? wide : narrow)) bn = 512;
  // Splitting K costs 1 to 2 us (the exchange, and clusters to place) and saves time by stage: over four CTAs it pays from eight stages on, as
  // far as the clusters run at once, over two from sixteen, or from 22 where there are tiles for more than a third of the SMs.  us with one / two /
  // four CTAs: 471x1672x1216 (56 tiles, 5 stages) 8.2 / 9.2 / -; 512x2048x2048 (64, 8) 8.9 / 10.6 / -; 93x1960x2560 (16, 10) 9.0 / 8.8 / 8.4;
  // 323x1536x7616 (36, 30; 36 clusters of four are more than run at once) 15.6 / 13.3 / 18.2; 152x2456x7168 (40, 28) 16.7 / 14.0 / -;
  // 320x2192x5760 (54, 23) 14.2 / 14.0 / -; 300x1024x8192 (24, 32) 15.9 / 12.5 / 12.3.
  split = 1;
  if (bn == 128 && stages >= 8) {
    const int64_t tiles = m128 * n128;
    if (tiles * 4 <= sms && tiles <= resident_splits_of_four()) split = 4;
    else if (tiles * 2 <= sms && stages >= (tiles * 3 <= sms ? 16 : 22)) split = 2;
  }
}

template <bool kGrouped>
int dispatch_gemm(int bn, const CUtensorMap& ma, const CUtensorMap& mb, const GemmParams& p, int max_m_tiles, cudaStream_t st,
                  const CUtensorMap* mo = nullptr) {
  if (bn == 256) return launch_gemm<256, kStageKb, kGrouped>(ma, mb, p, max_m_tiles, st, mo);
  return launch_gemm<128, kStageKb, kGrouped>(ma, mb, p, max_m_tiles, st);
}

}  // namespace
}  // namespace b200fp4

using namespace b200fp4;

extern "C" size_t b200fp4_gemm_workspace_bytes(int64_t M, int64_t N, int64_t K) {
  (void)M; (void)N; (void)K;
  return 256;
}

int b200fp4::dense_gemm_check(const void* a_codes, const void* b_codes, const void* sfa, const void* sfb, const float* alpha,
                              const void* out, int out_dtype, int64_t M, int64_t N, int64_t K, int tile_n, const void* workspace,
                              size_t workspace_bytes) {
  if (M < 0 || N <= 0 || K <= 0 || (K % 64) != 0) return B200FP4_STATUS_INVALID_VALUE;
  if (out_dtype != B200FP4_DTYPE_BF16 && out_dtype != B200FP4_DTYPE_F16 && out_dtype != B200FP4_DTYPE_F32)
    return B200FP4_STATUS_NOT_SUPPORTED;
  if (M == 0) return B200FP4_STATUS_SUCCESS;
  if (!a_codes || !b_codes || !sfa || !sfb || !alpha || !out) return B200FP4_STATUS_INVALID_VALUE;
  if (!aligned(a_codes, 16) || !aligned(b_codes, 16) || !aligned(sfa, 16) || !aligned(sfb, 16) || !aligned(out, 16) ||
      ((K / 2) % 16) != 0)
    return B200FP4_STATUS_INVALID_VALUE;
  if (!workspace || workspace_bytes < 256 || !aligned(workspace, 16)) return B200FP4_STATUS_ALLOC_FAILED;
  if (tile_n != 0 && tile_n != 128 && tile_n != 256 && tile_n != 512) return B200FP4_STATUS_INVALID_VALUE;
  if (tile_n == 512 && out_dtype == B200FP4_DTYPE_F32) return B200FP4_STATUS_NOT_SUPPORTED;
  if (M > (1 << 24) || N > (1 << 24) || K > (1 << 24)) return B200FP4_STATUS_NOT_SUPPORTED;
  return B200FP4_STATUS_SUCCESS;
}

// early_b: see GemmParams
static int gemm_nvfp4(const void* a_codes, const void* b_codes, const void* sfa, const void* sfb, const float* alpha, void* out,
                      int out_dtype, int64_t M, int64_t N, int64_t K, int tile_n, void* workspace, size_t workspace_bytes, void* stream,
                      bool early_b) {
  const int refused = dense_gemm_check(a_codes, b_codes, sfa, sfb, alpha, out, out_dtype, M, N, K, tile_n, workspace, workspace_bytes);
  if (refused != B200FP4_STATUS_SUCCESS || M == 0) return refused;
  if (b200fp4_has_hardware_acceleration() != 1) return B200FP4_STATUS_ARCH_MISMATCH;
  cudaStream_t st = (cudaStream_t)stream;
  if (tile_n == 0 && M <= kSmallMaxM) {
    const SmallPlan small = small_gemm_plan(M, N, K, stream_capturing(st) ? SmallUse::kCodesInGraph : SmallUse::kCodes);
    CUtensorMap mw;
    if (small.ok) {
      if (!make_map(&mw, b_codes, (uint64_t)N, (uint64_t)K / 2, kBM, kStageKb * 32)) return B200FP4_STATUS_INTERNAL_ERROR;
      return launch_gemm_small(small, mw, a_codes, 0, K, nullptr, reinterpret_cast<const uint8_t*>(sfa), reinterpret_cast<const uint8_t*>(sfb),
                               alpha, out, out_dtype, (int)M, (int)N, (int)K, reinterpret_cast<int*>(workspace), st);
    }
  }
  GemmParams p;
  p.sfa = reinterpret_cast<const uint8_t*>(sfa);
  p.sfb = reinterpret_cast<const uint8_t*>(sfb);
  p.alpha = alpha;
  p.out = out;
  p.out_bf16 = out_dtype == B200FP4_DTYPE_BF16;
  p.out_f32 = out_dtype == B200FP4_DTYPE_F32;
  p.M = (int)M; p.N = (int)N; p.K = (int)K;
  p.m_tiles = (int)((M + kBM - 1) / kBM);
  p.status = reinterpret_cast<int*>(workspace);
  p.early_b = early_b;
  int bn = tile_n, split = 1;
  if (bn == 0) pick_dense_tile(M, N, (K + 255) / 256, p.out_f32 != 0, bn, split);
  if (bn == 512) {
    // 256 x 256 tiles on CTA pairs (tcgen05 cta_group::2)
    CUtensorMap pa, pb;
    if (!make_map(&pa, a_codes, (uint64_t)M, (uint64_t)K / 2, 128, 128) ||
        !make_map(&pb, b_codes, (uint64_t)N, (uint64_t)K / 2, 128, 128))
      return B200FP4_STATUS_INTERNAL_ERROR;
    const int rc2 = launch_gemm_pair(pa, pb, p.sfa, p.sfb, alpha, out, p.out_bf16, (int)M, (int)N, (int)K, p.status, st);
    if (rc2 != B200FP4_STATUS_SUCCESS) return rc2;
    return finish_launch(1);
  }
  CUtensorMap ma, mb;
  if (!make_map(&ma, a_codes, (uint64_t)M, (uint64_t)K / 2, kBM, kStageKb * 32) ||
      !make_map(&mb, b_codes, (uint64_t)N, (uint64_t)K / 2, (uint32_t)bn, kStageKb * 32))
    return B200FP4_STATUS_INTERNAL_ERROR;
  p.g_hdr = nullptr;
  p.g_mtiles = nullptr;
  p.g_alphas = nullptr;
  p.g_sfb_expert_bytes = 0;
  // wide tiles, 16-bit output with 16-byte aligned rows: tiles leave through the copy engine
  CUtensorMap mo;
  const bool tma_out = bn == 256 && !p.out_f32 && (N % 8) == 0 && make_out_map(&mo, out, (uint64_t)M, (uint64_t)N);
  p.out_tma = tma_out ? 1 : 0;
  int rc = split == 4   ? launch_gemm<128, kStageKb, false, false, 4>(ma, mb, p, p.m_tiles, st)
           : split == 2 ? launch_gemm<128, kStageKb, false, false, 2>(ma, mb, p, p.m_tiles, st)
                        : dispatch_gemm<false>(bn, ma, mb, p, p.m_tiles, st, tma_out ? &mo : nullptr);
  if (rc != B200FP4_STATUS_SUCCESS) return rc;
  return finish_launch(1);
}

extern "C" int b200fp4_gemm_nvfp4(const void* a_codes, const void* b_codes, const void* sfa, const void* sfb,
                                  const float* alpha, void* out, int out_dtype, int64_t M, int64_t N, int64_t K,
                                  int tile_n, void* workspace, size_t workspace_bytes, void* stream) {
  return gemm_nvfp4(a_codes, b_codes, sfa, sfb, alpha, out, out_dtype, M, N, K, tile_n, workspace, workspace_bytes, stream, false);
}

// ---------------------------------------------------------------------------------------- linear layer in one call

// y = NVFP4(x) @ W^T: the activation quantizer and the GEMM queued by one call (two launches a few microseconds apart;
// through two Python calls the GPU idles between them for longer than either kernel runs at prefill sizes).
// workspace: [GEMM workspace (status word first) | codes M*K/2 | swizzled block scales], each part 256-byte aligned.
static size_t linear_part(size_t v) { return (v + 255) / 256 * 256; }

extern "C" size_t b200fp4_linear_workspace_bytes(int64_t M, int64_t N, int64_t K) {
  if (M < 0 || N <= 0 || K <= 0 || (K % 16) != 0) return 0;
  return linear_part((size_t)M * (size_t)K / 2) + linear_part(b200fp4_sf_swizzled_bytes(M, K / 16)) +
         linear_part(b200fp4_gemm_workspace_bytes(M, N, K));
}

extern "C" int b200fp4_linear_nvfp4(const void* x, int x_dtype, int64_t ldx, const float* x_global_scale, const void* w_codes,
                                    const void* w_sf, const float* alpha, void* out, int out_dtype, int64_t M, int64_t N,
                                    int64_t K, int tile_n, void* workspace, size_t workspace_bytes, void* stream) {
  if (M < 0 || N <= 0 || K <= 0 || (K % 64) != 0) return B200FP4_STATUS_INVALID_VALUE;
  if (M == 0) return B200FP4_STATUS_SUCCESS;
  if (!workspace || !aligned(workspace, 256) || workspace_bytes < b200fp4_linear_workspace_bytes(M, N, K))
    return B200FP4_STATUS_ALLOC_FAILED;
  const size_t gemm_bytes = b200fp4_gemm_workspace_bytes(M, N, K);
  unsigned char* gemm_ws = static_cast<unsigned char*>(workspace);
  unsigned char* codes = gemm_ws + linear_part(gemm_bytes);
  unsigned char* sf = codes + linear_part((size_t)M * (size_t)K / 2);
  // what either step would refuse, before the first is queued
  int rc = quantize_check(x, x_dtype, M, K, ldx, x_global_scale, codes, sf);
  if (rc == B200FP4_STATUS_SUCCESS)
    rc = dense_gemm_check(codes, w_codes, sf, w_sf, alpha, out, out_dtype, M, N, K, tile_n, gemm_ws, gemm_bytes);
  if (rc != B200FP4_STATUS_SUCCESS) return rc;
  if (b200fp4_has_hardware_acceleration() != 1) return B200FP4_STATUS_ARCH_MISMATCH;
  const bool captured = M > 16 && M <= kSmallMaxM && stream_capturing((cudaStream_t)stream);      // up to 16 tokens the plan is the same
  const SmallPlan small = small_gemm_plan(M, N, K, captured ? SmallUse::kLinearInGraph : SmallUse::kLinear);
  if (tile_n == 0 && small.ok) {
    // few tokens: quantized inside the GEMM
    CUtensorMap mw;
    if (!make_map(&mw, w_codes, (uint64_t)N, (uint64_t)K / 2, kBM, kStageKb * 32)) return B200FP4_STATUS_INTERNAL_ERROR;
    return launch_gemm_small(small, mw, x, x_dtype, ldx, x_global_scale, nullptr, reinterpret_cast<const uint8_t*>(w_sf), alpha, out, out_dtype,
                             (int)M, (int)N, (int)K, reinterpret_cast<int*>(gemm_ws), (cudaStream_t)stream);
  }
  rc = b200fp4_quantize(x, x_dtype, M, K, ldx, x_global_scale, codes, sf, 1, stream);
  if (rc != B200FP4_STATUS_SUCCESS) return rc;
  // The quantizer lets the GEMM start only after it has waited for everything before it: whatever wrote the weights is done.
  return gemm_nvfp4(codes, w_codes, sf, w_sf, alpha, out, out_dtype, M, N, K, tile_n, gemm_ws, gemm_bytes, stream, true);
}

// ---------------------------------------------------------------------------------------- grouped entry points

extern "C" size_t b200fp4_grouped_gemm_workspace_bytes(int64_t rows_capacity, int64_t E) {
  if (rows_capacity < 0 || E < 0) return 0;
  return 256 + (size_t)grouped_max_tiles(rows_capacity, E) * sizeof(int4);
}

namespace b200fp4 {

int grouped_gemm_check(const void* a_codes, const void* b_codes, const void* a_sf, const void* b_sf, const float* alphas,
                       const int32_t* expert_offsets, const int32_t* sf_offsets, const void* out, int out_dtype, int64_t rows_capacity,
                       int64_t N, int64_t K, int64_t E, int tile_n, const void* workspace, size_t workspace_bytes, const void* q_sf,
                       const float* q_gs, bool stage_sf) {
  const bool fused = q_sf != nullptr;
  if (stage_sf && !fused) return B200FP4_STATUS_INVALID_VALUE;
  if (fused && (!q_gs || (N % 256) != 0 || !aligned(out, 32) || !aligned(q_sf, 4))) return B200FP4_STATUS_INVALID_VALUE;
  if (rows_capacity < 0 || N <= 0 || K <= 0 || E <= 0 || (K % 64) != 0) return B200FP4_STATUS_INVALID_VALUE;
  if (out_dtype != B200FP4_DTYPE_BF16 && out_dtype != B200FP4_DTYPE_F16) return B200FP4_STATUS_NOT_SUPPORTED;
  if (rows_capacity == 0) return B200FP4_STATUS_SUCCESS;
  if (!a_codes || !b_codes || !a_sf || !b_sf || !alphas || !expert_offsets || !sf_offsets || !out)
    return B200FP4_STATUS_INVALID_VALUE;
  if (!aligned(a_codes, 16) || !aligned(b_codes, 16) || !aligned(a_sf, 16) || !aligned(b_sf, 16) || !aligned(out, 16) ||
      ((K / 2) % 16) != 0)
    return B200FP4_STATUS_INVALID_VALUE;
  if (E > kGroupMaxExperts || rows_capacity > (1 << 24) || N > (1 << 20) || K > (1 << 24) || E * N > (int64_t)1 << 30)
    return B200FP4_STATUS_NOT_SUPPORTED;
  if (tile_n != 0 && tile_n != 128 && tile_n != 256 && tile_n != 512) return B200FP4_STATUS_INVALID_VALUE;
  if (tile_n == 512 && out_dtype == B200FP4_DTYPE_F32) return B200FP4_STATUS_NOT_SUPPORTED;
  if (fused && tile_n == 128) return B200FP4_STATUS_INVALID_VALUE;
  if (!workspace || !aligned(workspace, 16) || workspace_bytes < b200fp4_grouped_gemm_workspace_bytes(rows_capacity, E))
    return B200FP4_STATUS_ALLOC_FAILED;
  return B200FP4_STATUS_SUCCESS;
}

int grouped_gemm(const void* a_codes, const void* b_codes, const void* a_sf, const void* b_sf, const float* alphas,
                 const int32_t* expert_offsets, const int32_t* sf_offsets, void* out, int out_dtype, int64_t rows_capacity, int64_t N,
                 int64_t K, int64_t E, int tile_n, void* workspace, size_t workspace_bytes, void* stream, void* q_sf, const float* q_gs,
                 bool tiles_ready, bool stage_sf) {
  const int refused = grouped_gemm_check(a_codes, b_codes, a_sf, b_sf, alphas, expert_offsets, sf_offsets, out, out_dtype, rows_capacity,
                                         N, K, E, tile_n, workspace, workspace_bytes, q_sf, q_gs, stage_sf);
  if (refused != B200FP4_STATUS_SUCCESS || rows_capacity == 0) return refused;
  if (b200fp4_has_hardware_acceleration() != 1) return B200FP4_STATUS_ARCH_MISMATCH;
  const bool fused = q_sf != nullptr;
  cudaStream_t st = (cudaStream_t)stream;
  const int max_tiles = grouped_max_tiles(rows_capacity, E);
  GemmParams p;
  p.sfa = reinterpret_cast<const uint8_t*>(a_sf);
  p.sfb = reinterpret_cast<const uint8_t*>(b_sf);
  p.alpha = nullptr;
  p.out = out;
  p.out_bf16 = out_dtype == B200FP4_DTYPE_BF16;
  p.out_f32 = 0;
  p.out_tma = 0;
  p.M = (int)rows_capacity; p.N = (int)N; p.K = (int)K;
  p.m_tiles = max_tiles;
  p.status = grouped_status(workspace);
  p.early_b = 0;
  p.g_hdr = grouped_hdr(workspace);
  p.g_mtiles = grouped_tiles(workspace);
  p.g_alphas = alphas;
  p.g_sfb_expert_bytes = (long long)b200fp4_sf_swizzled_bytes(N, K / 16);
  p.q_inter = fused ? (int)(N / 2) : 0;
  p.q_sf = reinterpret_cast<uint8_t*>(q_sf);
  p.q_gs = q_gs;
  // short K means short main loops: prefer the double-buffered narrow tile there, unless there are several
  // waves of wide tiles anyway (then halving the A re-reads and the tile count wins: 171 vs 183 us on
  // 81,920 rows x 2048 columns, K = 512)
  int bn = tile_n;
  if (bn == 0) {
    const long long wide_tiles = (long long)max_tiles * (N / 256);
    bn = (N % 256 == 0 && (K >= 2048 || wide_tiles >= 4LL * sm_count())) ? 256 : 128;
  }
  if (fused) bn = 256;
  CUtensorMap ma, mb;
  if (!make_map(&ma, a_codes, (uint64_t)rows_capacity, (uint64_t)K / 2, kBM, kStageKb * 32) ||
      !make_map(&mb, b_codes, (uint64_t)(E * N), (uint64_t)K / 2, fused ? 128u : (uint32_t)bn, kStageKb * 32))
    return B200FP4_STATUS_INTERNAL_ERROR;
  if (!tiles_ready)
    grouped_tiles_kernel<<<1, 1024, 0, st>>>(expert_offsets, sf_offsets, (int)E, grouped_hdr(workspace), grouped_tiles(workspace),
                                             max_tiles);
  int rc = stage_sf ? launch_gemm<256, kStageKb, true, true, 1, true>(ma, mb, p, max_tiles, st)
           : fused  ? launch_gemm<256, kStageKb, true, true>(ma, mb, p, max_tiles, st)
                    : dispatch_gemm<true>(bn, ma, mb, p, max_tiles, st);
  if (rc != B200FP4_STATUS_SUCCESS) return rc;
  return finish_launch(tiles_ready ? 1 : 2);
}

}  // namespace b200fp4

extern "C" int b200fp4_grouped_gemm_nvfp4(const void* a_codes, const void* b_codes, const void* a_sf, const void* b_sf,
                                          const float* alphas, const int32_t* expert_offsets, const int32_t* sf_offsets,
                                          void* out, int out_dtype, int64_t rows_capacity, int64_t N, int64_t K, int64_t E,
                                          int tile_n, void* workspace, size_t workspace_bytes, void* stream) {
  return grouped_gemm(a_codes, b_codes, a_sf, b_sf, alphas, expert_offsets, sf_offsets, out, out_dtype, rows_capacity, N, K, E, tile_n,
                      workspace, workspace_bytes, stream, nullptr, nullptr, false, false);
}

extern "C" int b200fp4_grouped_gemm_nvfp4_silu_quant(const void* a_codes, const void* b_codes, const void* a_sf,
                                                     const void* b_sf, const float* alphas, const int32_t* expert_offsets,
                                                     const int32_t* sf_offsets, const float* out_global_scales,
                                                     int mid_dtype, void* out_codes, void* out_sf, int64_t rows_capacity,
                                                     int64_t N, int64_t K, int64_t E, void* workspace,
                                                     size_t workspace_bytes, void* stream) {
  if (!out_sf || !out_global_scales) return B200FP4_STATUS_INVALID_VALUE;
  return grouped_gemm(a_codes, b_codes, a_sf, b_sf, alphas, expert_offsets, sf_offsets, out_codes, mid_dtype, rows_capacity, N, K, E, 0,
                      workspace, workspace_bytes, stream, out_sf, out_global_scales, false, false);
}

extern "C" int b200fp4_shuffle_rows(const void* in, int64_t row_bytes, const int32_t* dst2src, int64_t n_dst,
                                    int64_t src_div, void* out, void* stream) {
  if (n_dst < 0 || row_bytes <= 0 || (row_bytes % 16) != 0 || src_div <= 0) return B200FP4_STATUS_INVALID_VALUE;
  if (n_dst == 0) return B200FP4_STATUS_SUCCESS;
  if (!in || !dst2src || !out || !aligned(in, 16) || !aligned(out, 16)) return B200FP4_STATUS_INVALID_VALUE;
  const int64_t total = n_dst * (row_bytes / 16);
  int64_t blocks = (total + 255) / 256;
  if (blocks > 16 * (int64_t)sm_count()) blocks = 16 * (int64_t)sm_count();
  shuffle_rows_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(
      reinterpret_cast<const uint4*>(in), dst2src, (int)src_div, row_bytes / 16, n_dst, reinterpret_cast<uint4*>(out));
  return finish_launch(1);
}

