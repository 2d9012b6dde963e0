// Gate_up, SiLU and down projection of the 2:4-sparse MoE decode layer for few (token, expert) pairs, sm_100a.
//
// One or a few decoding tokens leave the layer's general kernel (sparse_moe.cu) a chain of waits: plan, records, weights, K-slices in
// turns of a ring, a fence and a counter in memory between the projections.  Here a cluster of blocks takes one pair from its expert
// id to its row of the down projection:
//   * no plan: a pair's expert comes straight from the ids; pairs that share an expert each stream its weights (once from HBM, then L2);
//   * K is split over all warps of a block, 16 of them, and the 128-column groups over the blocks, so that a warp has a handful of
//     32-wide steps of both projections; the weights of both are requested at once, as far as the ring holds them, before the
//     activations are even converted -- the down projection's do not depend on anything;
//   * SiLU(gate)*up goes to the other blocks of the cluster through distributed shared memory and a cluster barrier instead of memory,
//     fence and counter.
// Arithmetic as in the general kernel: E2M1 x E4M3 products exact in f16, mma.sp with f32 sums, f16 between the projections, f32 rows out.  The
// K-slices of a column are added in a fixed order: every fourth by one of four lanes, then those four sums by a butterfly.  The token's value stands in all eight columns of an mma; one is read.
#include "moe_small.cuh"

#include <math.h>

#include <mutex>

namespace b200fp4 {
namespace {

constexpr int kWarps = 16;
constexpr int kThreads = 32 * kWarps;
constexpr int kSlots = 4;                        // ring of a warp, in 32-wide steps of 128 columns: 115 KB in flight per SM
constexpr int kStage = 14 * 128;                 // 8 compressed, 4 metadata, 2 scale rows of 128 bytes
constexpr int kMaxCluster = 8;
constexpr int64_t kMaxWidth = 8192;              // H and I: activations of one token in shared memory, f16

struct SmallShape {
  int cluster;
  int ga, gb;          // 128-column groups per block of either projection
  int wa, wb;          // warps that share one of them
};

__host__ __device__ __forceinline__ size_t small_smem(int H, int I) {
  return 128 + (size_t)kWarps * kSlots * kStage + (size_t)kWarps * 512 + (size_t)(H + I) * 2;
}

// where the 16 bits of element k stand in the fragment order of its group of 32 (word 4i + t at 4t + i)
__device__ __forceinline__ uint32_t frag_byte(int k) {
  const int w = (k & 31) >> 1;
  return (uint32_t)(k >> 5) * 64u + (uint32_t)((w & 3) * 4 + (w >> 2)) * 4u + (uint32_t)(k & 1) * 2u;
}

template <bool kBf16>
__global__ void __launch_bounds__(kThreads, 1) moe_small_kernel(const MoeSmallArgs a, const SmallShape sh) {
  extern __shared__ unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane >> 2, t = lane & 3, fr = lane >> 3, fc = lane & 7;
  const int pair = (int)(blockIdx.x / (unsigned)sh.cluster), rank = (int)(blockIdx.x % (unsigned)sh.cluster);
  const uint32_t base = (shared_addr(smem_raw) + 127u) & ~127u;
  const uint32_t ring = base + (uint32_t)warp * (kSlots * kStage), part = base + kWarps * kSlots * kStage;
  const uint32_t xs = part + kWarps * 512, acts = xs + (uint32_t)a.H * 2;      // activations of either projection, fragment order
  const int H = a.H, I = a.I, N13 = 2 * I;
  // this warp's share: group, first step and number of steps (every wa-th / wb-th)
  const int ga_first = rank * sh.ga, ga_here = min(sh.ga, I / 64 - ga_first), gb_first = rank * sh.gb, gb_here = min(sh.gb, H / 128 - gb_first);
  const int a_group = warp / sh.wa, a_slice = warp - a_group * sh.wa, b_group = warp / sh.wb, b_slice = warp - b_group * sh.wb;
  const int n_a = a_group < ga_here ? (H / 32 - a_slice + sh.wa - 1) / sh.wa : 0;
  const int n_b = b_group < gb_here ? (I / 32 - b_slice + sh.wb - 1) / sh.wb : 0;
  // copies: lane (fr, fc) takes 16 columns of rows fr and fr + 4; chunks XOR-swizzled as in the general kernel (sparse_mma.cuh)
  const uint32_t d_comp = (uint32_t)fr * 128u + (uint32_t)((fc ^ (2 * (fr & 3))) << 4);
  const uint32_t d_meta = 1024u + (uint32_t)fr * 128u + (uint32_t)((fc ^ (4 * (fr >> 1))) << 4);
  const uint32_t d_scale = 1536u + (uint32_t)fr * 128u + (uint32_t)fc * 16u;
  const int grp_a = ga_first + a_group, grp_b = gb_first + b_group;
  const int col_a = fc < 4 ? grp_a * 64 + fc * 16 : I + grp_a * 64 + (fc - 4) * 16, col_b = grp_b * 128 + fc * 16;
  constexpr int kXLoads = (int)(kMaxWidth / 8 / kThreads);
  cluster_arrive();                                // the other blocks run before anything is sent to them; waited for further down
  pdl_wait();
  pdl_launch_dependents();
  const int m = pair / a.topk;
  const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(a.hidden) + (int64_t)m * a.ld_h);
  uint4 x[kXLoads];
#pragma unroll
  for (int i = 0; i < kXLoads; ++i)
    if (threadIdx.x + i * kThreads < H / 8) x[i] = src[threadIdx.x + i * kThreads];
  int e = a.ids[(int64_t)m * a.ids_ld + (pair - m * a.topk)];
  if (a.expert_map != nullptr) e = (e >= 0 && e < a.global_E) ? a.expert_map[e] : -1;
  if (e < 0 || e >= a.E) e = -1;
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.status = 0;
  if (e < 0) {                                     // the same for all blocks of the cluster
    cluster_wait();
    return;
  }
  // The stream of this warp's steps: those of the gate_up projection, then those of the down projection.  Where its next copies come from and
  // go to, and how far apart the steps of the projection lie; always one commit group a step, so that the wait counts stay fixed.
  struct Stream {
    const uint8_t *comp, *meta, *scale;
    int64_t comp_step, half;          // bytes between steps and between compressed rows 0 and 4 of one; metadata 1/2, scales 1/4 of that
    int left, then;                   // steps of this projection, of the next
    uint32_t slot;
  } f;
  auto start = [&](const SparseWeights& w, int N, int col, int first, int stride) {
    const int64_t lane_off = (int64_t)fr * N + col;
    f.comp = w.comp + (int64_t)e * w.comp_e + (int64_t)first * 8 * N + lane_off;
    f.meta = w.meta + (int64_t)e * w.meta_e + (int64_t)first * 4 * N + lane_off;
    f.scale = w.scale + (int64_t)e * w.scale_e + (int64_t)first * 2 * N + lane_off;
    f.comp_step = (int64_t)stride * 8 * N;
    f.half = (int64_t)4 * N;
  };
  start(a.w13, N13, col_a, a_slice, sh.wa);
  f.left = n_a;
  f.then = n_b;
  f.slot = ring;
  const uint32_t ring_end = ring + kSlots * kStage;
  auto fetch = [&]() {
    if (f.left == 0 && f.then > 0) {
      start(a.w2, H, col_b, b_slice, sh.wb);
      f.left = f.then;
      f.then = 0;
    }
    if (f.left > 0) {
      cp_async16_s(f.slot + d_comp, f.comp);
      cp_async16_s(f.slot + 512u + d_comp, f.comp + f.half);
      cp_async16_s(f.slot + d_meta, f.meta);
      if (lane < 16) cp_async16_s(f.slot + d_scale, f.scale);
      f.comp += f.comp_step;
      f.meta += f.comp_step >> 1;
      f.scale += f.comp_step >> 2;
      --f.left;
    }
    f.slot = f.slot + kStage == ring_end ? ring : f.slot + kStage;
    cp_async_commit();
  };
#pragma unroll 1
  for (int j = 0; j < kSlots; ++j) fetch();
  const float g13 = a.w13.g[e], g2 = a.w2.g[e];
  // the token's activations as f16 in fragment order
#pragma unroll
  for (int i = 0; i < kXLoads; ++i) {
    const int chunk = threadIdx.x + i * kThreads;
    if (chunk >= H / 8) break;
    uint32_t w[4] = {x[i].x, x[i].y, x[i].z, x[i].w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (kBf16) {
        const __half2 h = __float22half2_rn(__bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[k])));
        w[k] = *reinterpret_cast<const uint32_t*>(&h);
      }
      asm volatile("st.shared.b32 [%0], %1;" ::"r"(xs + frag_byte(8 * chunk + 2 * k)), "r"(w[k]) : "memory");
    }
  }
  __syncthreads();
  const uint32_t off_comp = (uint32_t)t * 128u + (uint32_t)((q ^ (2 * t)) << 4);
  const uint32_t off_meta = 1024u + (uint32_t)(2 * (t & 1)) * 128u + (uint32_t)((q ^ (4 * (t & 1))) << 4) + (uint32_t)(t >> 1) * 8u;
  const uint32_t off_scale = 1536u + (uint32_t)q * 16u;
  float acc[8][4];
  uint32_t st = ring;
  auto project = [&](uint32_t x, int stride, int n) {
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
#pragma unroll 1
    for (int s = 0; s < n; ++s, x += (uint32_t)stride * 64u) {
      cp_async_wait<kSlots - 1>();
      __syncwarp();
      WsStep w;
      w.v0 = lds128_at(st + off_comp);
      w.v1 = lds128_at(st + off_comp + 512u);
      w.m0 = lds64_at(st + off_meta);
      w.m1 = lds64_at(st + off_meta + 128u);
      w.s0 = lds128_at(st + off_scale);
      w.s1 = lds128_at(st + off_scale + 128u);
      w.b = lds128_at(x);
      __syncwarp();                                // all lanes have read the slot
      fetch();
      st = st + kStage == ring_end ? ring : st + kStage;
      ws_mma_step(acc, w);
    }
    // The sums of this warp's slice, 128 columns: column 2h + r of a quad's 16 is element 2r of mma kJ[h] in the quad's first lane.
    constexpr int kJ[8] = {0, 2, 4, 6, 1, 3, 5, 7};
    if (n > 0 && t == 0) {
#pragma unroll
      for (int h = 0; h < 8; h += 2)
        sts128f_at(part + (uint32_t)warp * 512u + (uint32_t)q * 64u + (uint32_t)h * 8u, acc[kJ[h]][0], acc[kJ[h]][2], acc[kJ[h + 1]][0],
                   acc[kJ[h + 1]][2]);
    }
    __syncthreads();
  };
  // The sum of a column's K-slices by four lanes (lane % 4 takes every fourth slice), known to all four.
  auto sum_of = [&](int group, int share, int used, int col) {
    float v = 0.f;
    for (int s = t; s < used; s += 4) v += __uint_as_float(lds32_at(part + (uint32_t)(group * share + s) * 512u + (uint32_t)col * 4u));
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    return v;
  };

  project(xs + (uint32_t)a_slice * 64u + (uint32_t)t * 16u, sh.wa, n_a);
  cluster_wait();
  {
    // a warp finishes four columns at a time: quads 0-3 sum the gate, 4-7 the up half
    const int used = min(sh.wa, H / 32);
    for (int i = warp; i < ga_here * 16; i += kWarps) {
      const int group = i >> 4, col = (i & 15) * 4 + (q & 3);
      const float v = sum_of(group, sh.wa, used, col + (q >> 2) * 64) * g13;
      const float up = __shfl_down_sync(0xffffffffu, v, 16);
      const float act = v / (1.0f + __expf(-v)) * up;                  // lanes 0..15
      const float next = __shfl_down_sync(0xffffffffu, act, 4);        // of the column after
      const __half2 h = __floats2half2_rn(act, next);
      // quads 0 and 2 hold two neighbouring columns, which go to the cluster's blocks
      if (lane < 16 && (q & 1) == 0) {
        const uint32_t at = acts + frag_byte((ga_first + group) * 64 + col);
        for (int r = t; r < sh.cluster; r += 4)
          asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(map_to_cta(at, (uint32_t)r)), "r"(*reinterpret_cast<const uint32_t*>(&h)) : "memory");
      }
    }
  }
  __syncwarp();
  cluster_arrive();
  cluster_wait();                                  // all of the token's activations are here, and the partial sums have been read
  project(acts + (uint32_t)b_slice * 64u + (uint32_t)t * 16u, sh.wb, n_b);
  {
    const int used = min(sh.wb, I / 32);
    for (int i = warp; i < gb_here * 16; i += kWarps) {
      const float v = sum_of(i >> 4, sh.wb, used, (i & 15) * 8 + q) * g2;
      if (t == 0) a.down[(int64_t)pair * H + (int64_t)gb_first * 128 + i * 8 + q] = v;
    }
  }
  cp_async_wait<0>();
}

SmallShape shape_for(int cluster, int64_t H, int64_t I) {
  SmallShape s;
  s.cluster = cluster;
  s.ga = (int)((I / 64 + cluster - 1) / cluster);
  s.gb = (int)((H / 128 + cluster - 1) / cluster);
  s.wa = kWarps / s.ga;
  s.wb = kWarps / s.gb;
  return s;
}

template <bool kBf16>
bool prepare() {
  static std::once_flag once[64];
  static bool ok[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  std::call_once(once[dev], [&] {
    ok[dev] = cudaFuncSetAttribute(moe_small_kernel<kBf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)small_smem(kMaxWidth, kMaxWidth)) ==
              cudaSuccess;
    if (!ok[dev]) cudaGetLastError();
  });
  return ok[dev];
}

// Clusters of c blocks that run at once
int resident_pairs(int c) {
  static ResidentClusters counts[kMaxCluster + 1][64];
  return resident_clusters_of(counts[c], moe_small_kernel<true>, c, kThreads, small_smem(kMaxWidth, kMaxWidth));
}

}  // namespace

// The cluster size that is expected to take the least time, if that is less than on the general path.  `local` of the P pairs are expected to
// have an expert here (fewer than P on an expert-parallel rank); the clusters of the others leave when they have seen their id.  Those that
// stay, twice the standard deviation above the expected number, run at once; where all P do not, each further round of them is 2.37 us.
// Times fitted to B200, us per layer (pairs, H, I: general / here, blocks per pair):
//   10, 2048, 512: 15.1 / 10.4, 8     20: 19.3 / 14.1, 6     40: 25.9 / 18.8, 3     60: 30.5 / 22.2, 2     140: 42.8 / 38.9, 1
//   24, 4096, 1024: 36.9 / 34.2, 4    64, 4096, 1024: 61.3 / 61.6, 2
// and of 512 experts on 8 ranks, 2048, 512: 10: 10.4 / 7.7, 8     40: 12.7 / 12.6, 8     100: 15.5 / 18.2, 4     140: 18.1 / 21.4, 4
// A block's time here is its warps' steps (one of all 16 warps takes 0.566 us: instruction issue) and 5.7 us.  The general path spreads all steps
// evenly over the SMs; a few pairs take their time in its chain of launches and loads.  Over 220 sizes, 1 to 8 ranks, the choice takes 1.2 % more
// than the best of all, 15 % at most, and 9 % at most more than the general path.
// Only the number of pairs is known here.  Tokens that route alike stream an expert once each, where the general path reads it once for
// eight: 12 tokens on the same ten of 512 experts 36.4 us here, 21.3 there, two by two alike 36.8 and 33.1, all different 37.6 and 40.9.
int moe_small_cluster(int64_t P, double local, int64_t H, int64_t I) {
  if (P < 1 || local <= 0 || H > kMaxWidth || I > kMaxWidth) return 0;
  const double most = local + 2.0 * sqrt(local * (1.0 - local / (double)P));
  int best = 0;
  double here = 0;
  for (int c = 1; c <= kMaxCluster; ++c) {
    const SmallShape s = shape_for(c, H, I);
    if (s.ga > kWarps || s.gb > kWarps || most * c > sm_count() || most > resident_pairs(c)) continue;
    const int64_t steps = (H / 32 + s.wa - 1) / s.wa + (I / 32 + s.wb - 1) / s.wb;       // of a warp
    const double rounds = (double)P / resident_pairs(c) - 1.0, t = 5.66 + 0.566 * (double)steps + (rounds > 0 ? 2.37 * rounds : 0.0);
    if (best == 0 || t < here) {
      best = c;
      here = t;
    }
  }
  const double all = local * (double)(H / 32) * (double)(I / 32) * 0.75;                  // steps of both projections: H/32 I/64 + I/32 H/128
  const double width = (double)((H + I) / 32), general = 9.5 + 0.00025 * all + (0.0143 + 0.0033 * (local < 20 ? local : 20.0)) * width;
  return best > 0 && here < general ? best : 0;
}

int launch_moe_small(int cluster, bool bf16, const MoeSmallArgs& a, int64_t P, cudaStream_t st) {
  if (!(bf16 ? prepare<true>() : prepare<false>())) return B200FP4_STATUS_EXECUTION_FAILED;
  if (launch_pdl_cluster(cluster, bf16 ? moe_small_kernel<true> : moe_small_kernel<false>, dim3((unsigned)(P * cluster)), dim3(kThreads),
                         small_smem(a.H, a.I), st, a, shape_for(cluster, a.H, a.I)) != cudaSuccess) {
    cudaGetLastError();
    return B200FP4_STATUS_EXECUTION_FAILED;
  }
  return B200FP4_STATUS_SUCCESS;
}

}  // namespace b200fp4
