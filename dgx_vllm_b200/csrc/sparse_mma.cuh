// Low-level pieces shared by the 2:4-sparse tensor-core kernels: asynchronous copies, shared-memory loads, format decode,
// mma.sp, and the ring-stage geometry of the kernels whose warps own whole 128-column strips.
#pragma once

#include "common.cuh"

namespace b200fp4 {

// Where one projection's weights live.  Row r of the compressed tensor for expert e and column n:
//   comp  + e*comp_e  + (r/2)*comp_pair + (r&1)*comp_odd + n
//   meta  + e*meta_e  + (r/2)*meta_row + n            (one metadata row per two compressed rows)
//   scale + e*scale_e + srow*scale_row + n
// which covers both the separate tensors (sparse_fp4_v7.cu:158-167) and the interleaved
// [E, K/8, 4N] tensor (sparse_fp4_v7.cu:246-251).
struct SparseWeights {
  const uint8_t* comp;
  const uint8_t* meta;
  const uint8_t* scale;
  const float* g;
  int64_t comp_e, comp_pair, comp_odd;
  int64_t meta_e, meta_row;
  int64_t scale_e, scale_row;
};

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ uint32_t word_of(const uint4& v, int q) {
  return q == 0 ? v.x : (q == 1 ? v.y : (q == 2 ? v.z : v.w));
}
__device__ __forceinline__ __half2 as_h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }
__device__ __forceinline__ uint32_t shared_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t lds32_at(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint2 lds64_at(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint4 lds128_at(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float4 lds128f_at(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts64f_at(uint32_t a, float x, float y) {
  asm volatile("st.shared.v2.f32 [%0], {%1,%2};" ::"r"(a), "f"(x), "f"(y) : "memory");
}
__device__ __forceinline__ void sts128f_at(uint32_t a, float x, float y, float z, float w) {
  asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(a), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}
__device__ __forceinline__ void cp_async16_s(uint32_t smem_dst, const void* gmem_src) {
  asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(smem_dst), "l"(gmem_src) : "memory");
}

template <int SEL>
__device__ __forceinline__ void mma_sp_m16n8k32(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                const uint32_t (&b)[4], uint32_t e) {
  asm volatile(
      "mma.sp::ordered_metadata.sync.aligned.m16n8k32.row.col.f32.f16.f16.f32 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9,%10,%11}, {%0,%1,%2,%3}, %12, %13;"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(e), "n"(SEL));
}

// byte B of a word holds two E2M1 values -> half2 (low nibble in the low half)
template <int B>
__device__ __forceinline__ __half2 e2m1x2_to_h2(uint32_t w) {
  uint32_t r;
  if (B == 0) asm("{ .reg .b8 b0, b1, b2, b3; mov.b32 {b0, b1, b2, b3}, %1; cvt.rn.f16x2.e2m1x2 %0, b0; }" : "=r"(r) : "r"(w));
  else if (B == 1) asm("{ .reg .b8 b0, b1, b2, b3; mov.b32 {b0, b1, b2, b3}, %1; cvt.rn.f16x2.e2m1x2 %0, b1; }" : "=r"(r) : "r"(w));
  else if (B == 2) asm("{ .reg .b8 b0, b1, b2, b3; mov.b32 {b0, b1, b2, b3}, %1; cvt.rn.f16x2.e2m1x2 %0, b2; }" : "=r"(r) : "r"(w));
  else asm("{ .reg .b8 b0, b1, b2, b3; mov.b32 {b0, b1, b2, b3}, %1; cvt.rn.f16x2.e2m1x2 %0, b3; }" : "=r"(r) : "r"(w));
  return as_h2(r);
}
// half H (16 bits) of a word holds two E4M3 values -> half2
template <int H>
__device__ __forceinline__ __half2 e4m3x2_to_h2(uint32_t w) {
  uint32_t r;
  if (H == 0) asm("{ .reg .b16 lo, hi; mov.b32 {lo, hi}, %1; cvt.rn.f16x2.e4m3x2 %0, lo; }" : "=r"(r) : "r"(w));
  else asm("{ .reg .b16 lo, hi; mov.b32 {lo, hi}, %1; cvt.rn.f16x2.e4m3x2 %0, hi; }" : "=r"(r) : "r"(w));
  return as_h2(r);
}

constexpr int kWsStages = 4;
constexpr int kWsWarps = 16;
constexpr int kWsStageBytes = 14 * 128 + 512;     // 8 compressed + 4 metadata + 2 scale rows of 128 bytes, B fragments of 8 tokens

// Lane-constant shared-memory offsets of the warp-scheduled kernel.
// Stage layout: compressed rows 0..7 | metadata rows 0..3 | scale rows 0..1 (128 bytes each) | B fragments.  The 16-byte
// chunks of a compressed row r sit at chunk ^ 2(r%4), those of a metadata row at chunk ^ 4(r/2), so that the fragment
// loads (rows t and t+4 for lane t of a quad; metadata rows 2(t%2), 2(t%2)+1) spread over all banks.
struct WsLane {
  uint32_t ring;                                   // this warp's ring
  uint32_t d_comp, d_meta, d_scale, d_b;           // where this lane's copies land (compressed rows fr and fr+4, metadata / scale row fr)
  uint32_t off_comp, off_meta, off_scale;          // where its fragments are read from
  int lane, q, t, fr, fc;
};

template <int kS = kWsStages>
__device__ __forceinline__ WsLane ws_lane(unsigned char* smem) {
  WsLane L;
  L.lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  L.q = L.lane >> 2;
  L.t = L.lane & 3;
  L.fr = L.lane >> 3;
  L.fc = L.lane & 7;
  L.ring = ((shared_addr(smem) + 127u) & ~127u) + (uint32_t)warp * (kS * kWsStageBytes);
  L.d_comp = (uint32_t)L.fr * 128u + (uint32_t)((L.fc ^ (2 * (L.fr & 3))) << 4);
  L.d_meta = 1024u + (uint32_t)L.fr * 128u + (uint32_t)((L.fc ^ (4 * (L.fr >> 1))) << 4);
  L.d_scale = 1536u + (uint32_t)L.fr * 128u + (uint32_t)L.fc * 16u;
  L.d_b = 1792u + (uint32_t)L.lane * 16u;
  L.off_comp = (uint32_t)L.t * 128u + (uint32_t)((L.q ^ (2 * L.t)) << 4);
  L.off_meta = 1024u + (uint32_t)(2 * (L.t & 1)) * 128u + (uint32_t)((L.q ^ (4 * (L.t & 1))) << 4) + (uint32_t)(L.t >> 1) * 8u;
  L.off_scale = 1536u + (uint32_t)L.q * 16u;
  return L;
}

// What one lane reads of a ring stage (a 32-wide k-step of 128 columns) ...
struct WsStep {
  uint4 v0, v1;      // compressed rows t and t + 4 of the quad's 16 columns
  uint2 m0, m1;      // metadata rows 2(t%2), 2(t%2)+1
  uint4 s0, s1;      // block scales
  uint4 b;           // B fragments
};
__device__ __forceinline__ WsStep ws_load_step(const WsLane& L, uint32_t st) {
  WsStep w;
  w.v0 = lds128_at(st + L.off_comp);
  w.v1 = lds128_at(st + L.off_comp + 512u);
  w.m0 = lds64_at(st + L.off_meta);
  w.m1 = lds64_at(st + L.off_meta + 128u);
  w.s0 = lds128_at(st + L.off_scale);
  w.s1 = lds128_at(st + L.off_scale + 128u);
  w.b = lds128_at(st + L.d_b);
  return w;
}
// ... and its eight mma.sp: mma j takes columns 2h, 2h+1 of every quad as its rows q and q+8: bytes (2hf, 2hf+1) of word wi
// of the loaded vectors.  Even j: metadata from lanes t = 0, 1 (first half of the quad's columns), odd j: t = 2, 3.
__device__ __forceinline__ void ws_mma_step(float (&acc)[8][4], const WsStep& w) {
  const uint32_t bf[4] = {w.b.x, w.b.y, w.b.z, w.b.w};
  uint32_t em[4];
  em[0] = prmt(w.m0.x, w.m1.x, 0x5140u);
  em[1] = prmt(w.m0.x, w.m1.x, 0x7362u);
  em[2] = prmt(w.m0.y, w.m1.y, 0x5140u);
  em[3] = prmt(w.m0.y, w.m1.y, 0x7362u);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    constexpr int kH[8] = {0, 4, 1, 5, 2, 6, 3, 7};
    const int h = kH[j];
    const int wi = h >> 1, hf = h & 1;
    const uint32_t c0 = word_of(w.v0, wi), c1 = word_of(w.v1, wi);
    const __half2 sc0 = hf ? e4m3x2_to_h2<1>(word_of(w.s0, wi)) : e4m3x2_to_h2<0>(word_of(w.s0, wi));
    const __half2 sc1 = hf ? e4m3x2_to_h2<1>(word_of(w.s1, wi)) : e4m3x2_to_h2<0>(word_of(w.s1, wi));
    const __half2 a0 = __hmul2(hf ? e2m1x2_to_h2<2>(c0) : e2m1x2_to_h2<0>(c0), __low2half2(sc0));
    const __half2 a1 = __hmul2(hf ? e2m1x2_to_h2<3>(c0) : e2m1x2_to_h2<1>(c0), __high2half2(sc0));
    const __half2 a2 = __hmul2(hf ? e2m1x2_to_h2<2>(c1) : e2m1x2_to_h2<0>(c1), __low2half2(sc1));
    const __half2 a3 = __hmul2(hf ? e2m1x2_to_h2<3>(c1) : e2m1x2_to_h2<1>(c1), __high2half2(sc1));
    if ((j & 1) == 0)
      mma_sp_m16n8k32<0>(acc[j], *reinterpret_cast<const uint32_t*>(&a0), *reinterpret_cast<const uint32_t*>(&a1),
                         *reinterpret_cast<const uint32_t*>(&a2), *reinterpret_cast<const uint32_t*>(&a3), bf, em[j >> 1]);
    else
      mma_sp_m16n8k32<1>(acc[j], *reinterpret_cast<const uint32_t*>(&a0), *reinterpret_cast<const uint32_t*>(&a1),
                         *reinterpret_cast<const uint32_t*>(&a2), *reinterpret_cast<const uint32_t*>(&a3), bf, em[j >> 1]);
  }
}

}  // namespace b200fp4
