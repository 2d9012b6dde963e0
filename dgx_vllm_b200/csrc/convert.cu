// NVFP4 checkpoint layout -> 2:4 compressed layout of the sparse GEMV, on the GPU.
//
// Replaces the load-time Python loop of the reference (unpack_fp4_nibbles, apply_2of4_sparsity_fast,
// convert_expert_to_v7_gpu, convert_weight_batch_to_v7: sparse_fp4_kernel/sparse_v7_moe_patch.py:39-129),
// which runs torch.topk per expert for 512 experts x 48 layers.  In every group of four consecutive k the two codes of
// largest magnitude are kept; among equal magnitudes the LOWER index wins (torch.topk leaves that order unspecified, this
// rule is deterministic), and the kept indices are stored ascending.
// Outputs are transposed so that N is contiguous: comp_T [E, K/4, N], meta_T [E, K/8, N],
// scale_T [E, G, N] (plain transpose of the [E, N, G] block scales).
#include "common.cuh"

namespace b200fp4 {
namespace {

// Both tensors go through tiles of 128 rows n x 32 words of the source, read along k and stored along n, so that every
// global access is part of a whole 128-byte line on both sides.  One thread handles one word column of 16 rows, whose
// results are 16 neighbouring bytes of every output row.
// The copies (1 byte in and out per weight) would take 164 us for 512 experts of 1024 x 2048 codes and scales at the
// measured copy rate; the integer pipe is the other bound: deciding the two kept codes with packed comparisons costs 12
// integer instructions per group of four and measured 263 us, one thread per 4-byte word reading down a column of rows
// 1620 us.  So the decision is a lookup: the 12 magnitude bits of a group index a table in shared memory (three to four
// bank conflicts per warp on random codes) and six instructions per group are left.  Measured 231 us (codes 207, scales 24).
constexpr int kTileN = 128;
constexpr int kTileW = 32;
constexpr int kConvThreads = 256;
constexpr int kTableEntries = 4096;

// Metadata nibble i0 | i1 << 2 of a group whose magnitudes (low three bits of the E2M1 codes: 0, .5, 1, 1.5, 2, 3, 4, 6
// are increasing) are the four 3-bit fields of `mags`.
__device__ __forceinline__ uint32_t top2_of4(uint32_t mags) {
  uint32_t mag[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) mag[j] = (mags >> (3 * j)) & 7u;
  int a = 0;
#pragma unroll
  for (int j = 1; j < 4; ++j)
    if (mag[j] > mag[a]) a = j;
  int b = -1;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (j == a) continue;
    if (b < 0 || mag[j] > mag[b]) b = j;
  }
  return (uint32_t)(a < b ? a : b) | ((uint32_t)(a < b ? b : a) << 2);
}

// Table entries of the low group (first half of the table) and of the high group of a word: bits 0-7 (8-15) are the two
// byte selectors of the kept nibbles among the bytes of {word, word >> 4}, whose low halves are nibbles 0, 2, 4, 6 | 1, 3,
// 5, 7; bits 16-19 (20-23) the metadata nibble.  The entries of both groups OR together into what a word needs.
__device__ __forceinline__ uint32_t group_entry(uint32_t meta, bool high) {
  const uint32_t i0 = meta & 3u, i1 = meta >> 2, base = high ? 2u : 0u;
  const uint32_t s0 = (i0 >> 1) + ((i0 & 1u) << 2) + base, s1 = (i1 >> 1) + ((i1 & 1u) << 2) + base;
  return high ? (s0 << 8) | (s1 << 12) | (meta << 20) : s0 | (s1 << 4) | (meta << 16);
}

// The words of four rows at one word column -> two compressed rows and one metadata row of four columns each.
__device__ __forceinline__ void convert_words(const uint4& v, const unsigned char* table, uint32_t& comp0, uint32_t& comp1,
                                              uint32_t& meta) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  uint32_t c[4], x[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const uint32_t t = (w[r] & 0x07070707u) | ((w[r] >> 1) & 0x38383838u);      // six magnitude bits per byte
    const uint32_t u = ((t * 4u) & 0x00FC00FCu) | (t & ~0x00FC00FCu & 0x3F003F00u);    // 12 per half, times four
    x[r] = *reinterpret_cast<const uint32_t*>(table + (u & 0xFFFFu)) |
           *reinterpret_cast<const uint32_t*>(table + 4 * kTableEntries + (u >> 16));
    // the four kept nibbles, each in the low half of a byte (what stands in the upper halves is cut away)
    const uint32_t k = prmt(w[r], w[r] >> 4, x[r]);
    c[r] = (k & 0x000F000Fu) | ((k >> 4) & ~0x000F000Fu);                       // bytes 0 and 2: the two groups
  }
  const uint32_t t = prmt(c[0], c[1], 0x6240u), u = prmt(c[2], c[3], 0x6240u);
  comp0 = prmt(t, u, 0x5410u);
  comp1 = prmt(t, u, 0x7632u);
  meta = prmt(prmt(x[0], x[1], 0x0062u), prmt(x[2], x[3], 0x0062u), 0x5410u);
}

// sixteen consecutive bytes of an output row; kVec: N and the outputs are multiples of 16
template <bool kVec>
__device__ __forceinline__ void store16(uint8_t* dst, const uint32_t (&v)[4], int left) {
  if (kVec) {
    *reinterpret_cast<uint4*>(dst) = make_uint4(v[0], v[1], v[2], v[3]);
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (i < left) dst[i] = (uint8_t)(v[i >> 2] >> (8 * (i & 3)));
  }
}

// kScales false: src = codes [E, N, src_bytes], out0 = comp_T [E, src_bytes / 2, N], out1 = meta_T [E, src_bytes / 4, N].
// kScales true:  src = scales [E, N, src_bytes], out0 = scale_T [E, src_bytes, N].
// kVec: rows of whole 16-byte chunks on both sides and 16-byte aligned tensors; otherwise bytes are loaded and stored.
template <bool kScales, bool kVec>
__global__ void __launch_bounds__(kConvThreads, 4)
    convert_tile_kernel(const uint8_t* __restrict__ src, int N, int src_bytes, uint32_t n_tiles, uint32_t tiles_n, uint32_t tiles_e,
                        uint8_t* __restrict__ out0, uint8_t* __restrict__ out1) {
  extern __shared__ __align__(16) unsigned char smem[];
  // word-major; four rows are a 16-byte group, and group q of a word column sits at position q ^ (q / 8) % 4 ^ (chunk of the
  // column): then neither the stores of a loaded chunk (eight chunks x four rows per warp) nor the 16-byte reads (eight
  // neighbouring lanes read every fourth group) meet a bank twice
  uint32_t* tile = reinterpret_cast<uint32_t*>(smem);
  unsigned char* table = smem + 4 * kTileW * kTileN;
  const int words = (src_bytes + 3) >> 2;
  if (!kScales) {
    for (int i = threadIdx.x; i < kTableEntries; i += kConvThreads) {
      const uint32_t meta = top2_of4(i);
      reinterpret_cast<uint32_t*>(table)[i] = group_entry(meta, false);
      reinterpret_cast<uint32_t*>(table)[kTableEntries + i] = group_entry(meta, true);
    }
  }
  const int lc = threadIdx.x & 7, lrow = threadIdx.x >> 3;       // load: 16-byte chunk and row
  const int g = threadIdx.x & 7, wl = threadIdx.x >> 3;          // convert: group of 16 rows and word column
  uint4 v[4];
  struct Pos {
    uint32_t e, tw, tn;
  };
  auto pos_of = [&](uint32_t t) {      // tile -> expert, tile of words, tile of rows (fastest)
    Pos p;
    p.e = t / tiles_e;
    const uint32_t r = t - p.e * tiles_e;
    p.tw = r / tiles_n;
    p.tn = r - p.tw * tiles_n;
    return p;
  };
  auto load = [&](const Pos& at) {
    const int row = (int)at.tn * kTileN + lrow, b = ((int)at.tw * kTileW + lc * 4) * 4;
    const uint8_t* p = src + ((int64_t)at.e * N + row) * (int64_t)src_bytes + b;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[i] = make_uint4(0, 0, 0, 0);
      if (row + i * 32 < N && b < src_bytes) {
        if (kVec) {
          v[i] = ldg_stream_u4(p + (int64_t)(i * 32) * src_bytes);
        } else {
          uint32_t x[4] = {0, 0, 0, 0};
          for (int k = 0; k < 16; ++k)
            if (b + k < src_bytes) x[k >> 2] |= (uint32_t)p[(int64_t)(i * 32) * src_bytes + k] << (8 * (k & 3));
          v[i] = make_uint4(x[0], x[1], x[2], x[3]);
        }
      }
    }
  };
  Pos cur = pos_of(blockIdx.x);
  load(cur);
  for (uint32_t t = blockIdx.x; t < n_tiles; t += gridDim.x) {
    __syncthreads();             // the tile of the round before has been read (first round: the table is written below this)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int q = 8 * i + (lrow >> 2);
      uint32_t* d = tile + lc * 4 * kTileN + (((q ^ i ^ lc) << 2) | (lrow & 3));
      d[0] = v[i].x;
      d[kTileN] = v[i].y;
      d[2 * kTileN] = v[i].z;
      d[3 * kTileN] = v[i].w;
    }
    __syncthreads();
    const int64_t e = cur.e;
    const int w = (int)cur.tw * kTileW + wl, n = (int)cur.tn * kTileN + 16 * g, left = N - n;
    if (t + gridDim.x < n_tiles) {
      cur = pos_of(t + gridDim.x);
      load(cur);                 // in flight during the conversion of this tile
    }
    if (left <= 0 || w >= words) continue;
    uint32_t r0[4], r1[4], r2[4], r3[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int q = (4 * g + j) ^ ((g >> 1) & 3) ^ (wl >> 2);
      const uint4 x = *reinterpret_cast<const uint4*>(&tile[wl * kTileN + 4 * q]);
      if (kScales) {
        // 4 x 4 byte transpose: byte k of the four rows' words
        const uint32_t a = prmt(x.x, x.y, 0x5140u), b = prmt(x.x, x.y, 0x7362u);
        const uint32_t d = prmt(x.z, x.w, 0x5140u), f = prmt(x.z, x.w, 0x7362u);
        r0[j] = prmt(a, d, 0x5410u);
        r1[j] = prmt(a, d, 0x7632u);
        r2[j] = prmt(b, f, 0x5410u);
        r3[j] = prmt(b, f, 0x7632u);
      } else {
        convert_words(x, table, r0[j], r1[j], r2[j]);
      }
    }
    if (kScales) {
      uint8_t* dst = out0 + (e * src_bytes + 4 * w) * N + n;
      store16<kVec>(dst, r0, left);
      if (kVec || 4 * w + 1 < src_bytes) store16<kVec>(dst + N, r1, left);
      if (kVec || 4 * w + 2 < src_bytes) store16<kVec>(dst + 2 * (int64_t)N, r2, left);
      if (kVec || 4 * w + 3 < src_bytes) store16<kVec>(dst + 3 * (int64_t)N, r3, left);
    } else {
      const int64_t row = e * words + w;
      uint8_t* dst = out0 + 2 * row * N + n;
      store16<kVec>(dst, r0, left);
      store16<kVec>(dst + N, r1, left);
      store16<kVec>(out1 + row * N + n, r2, left);
    }
  }
}

template <bool kScales, bool kVec>
void launch_convert_t(const uint8_t* src, int64_t E, int64_t N, int64_t src_bytes, uint8_t* out0, uint8_t* out1, cudaStream_t st) {
  constexpr size_t smem = 4 * kTileW * kTileN + (kScales ? 0 : 2 * 4 * kTableEntries);
  static_assert(smem <= 48 * 1024, "four blocks per SM, no opt-in");
  const int64_t tiles_n = (N + kTileN - 1) / kTileN, tiles_w = (src_bytes + 4 * kTileW - 1) / (4 * kTileW);
  const int64_t n_tiles = E * tiles_n * tiles_w, most = 4 * (int64_t)sm_count();
  convert_tile_kernel<kScales, kVec><<<(unsigned)(n_tiles < most ? n_tiles : most), kConvThreads, smem, st>>>(
      src, (int)N, (int)src_bytes, (uint32_t)n_tiles, (uint32_t)tiles_n, (uint32_t)(tiles_n * tiles_w), out0, out1);
}

template <bool kScales>
void launch_convert(const uint8_t* src, int64_t E, int64_t N, int64_t src_bytes, uint8_t* out0, uint8_t* out1, cudaStream_t st) {
  if (src_bytes % 16 == 0 && N % 16 == 0 && aligned(src, 16) && aligned(out0, 16) && aligned(out1, 16))
    launch_convert_t<kScales, true>(src, E, N, src_bytes, out0, out1, st);
  else
    launch_convert_t<kScales, false>(src, E, N, src_bytes, out0, out1, st);
}

}  // namespace
}  // namespace b200fp4

using namespace b200fp4;

extern "C" int b200fp4_convert_to_sparse_2of4(const uint8_t* codes, const uint8_t* scales, int64_t E, int64_t N, int64_t K,
                                              int64_t G, uint8_t* comp_T, uint8_t* meta_T, uint8_t* scale_T, void* stream) {
  if (E <= 0 || N <= 0 || K <= 0 || (K % 8) != 0 || G <= 0) return B200FP4_STATUS_INVALID_VALUE;
  if (!codes || !comp_T || !meta_T || !aligned(codes, 4)) return B200FP4_STATUS_INVALID_VALUE;
  if ((scales == nullptr) != (scale_T == nullptr)) return B200FP4_STATUS_INVALID_VALUE;
  if (E > 65535 || K / 8 > 65535 || N > (1 << 24) || (scales && (G + 31) / 32 > 65535)) return B200FP4_STATUS_NOT_SUPPORTED;
  cudaStream_t st = (cudaStream_t)stream;
  launch_convert<false>(codes, E, N, K / 2, comp_T, meta_T, st);
  int launches = 1;
  if (scales) {
    launch_convert<true>(scales, E, N, G, scale_T, nullptr, st);
    ++launches;
  }
  return finish_launch(launches);
}
