// A block of 16 activations to NVFP4: what the stand-alone quantizer and the kernels that quantize their own operand share, so
// that all of them produce the same bytes.
#pragma once

#include "common.cuh"

namespace b200fp4 {

// Packed helpers on two 16-bit floats in one register.
template <typename T>
struct Pk;
template <>
struct Pk<__nv_bfloat16> {
  static __device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) {
    const __nv_bfloat162 r = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
    return *reinterpret_cast<const uint32_t*>(&r);
  }
  static __device__ __forceinline__ uint32_t absmax2(uint32_t a, uint32_t b) {
    const __nv_bfloat162 r = __hmax2(__habs2(*reinterpret_cast<const __nv_bfloat162*>(&a)), __habs2(*reinterpret_cast<const __nv_bfloat162*>(&b)));
    return *reinterpret_cast<const uint32_t*>(&r);
  }
  static __device__ __forceinline__ float lo(uint32_t w) { return __uint_as_float(w << 16); }
  static __device__ __forceinline__ float hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }
};
template <>
struct Pk<__half> {
  static __device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) {
    const __half2 r = __hmax2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
    return *reinterpret_cast<const uint32_t*>(&r);
  }
  static __device__ __forceinline__ uint32_t absmax2(uint32_t a, uint32_t b) {
    const __half2 r = __hmax2(__habs2(*reinterpret_cast<const __half2*>(&a)), __habs2(*reinterpret_cast<const __half2*>(&b)));
    return *reinterpret_cast<const uint32_t*>(&r);
  }
  static __device__ __forceinline__ float lo(uint32_t w) { return __low2float(*reinterpret_cast<const __half2*>(&w)); }
  static __device__ __forceinline__ float hi(uint32_t w) { return __high2float(*reinterpret_cast<const __half2*>(&w)); }
};

template <typename T>
__device__ __forceinline__ void unpack8(const uint4& raw, float* v) {
  v[0] = Pk<T>::lo(raw.x); v[1] = Pk<T>::hi(raw.x); v[2] = Pk<T>::lo(raw.y); v[3] = Pk<T>::hi(raw.y);
  v[4] = Pk<T>::lo(raw.z); v[5] = Pk<T>::hi(raw.z); v[6] = Pk<T>::lo(raw.w); v[7] = Pk<T>::hi(raw.w);
}

// max |x| over the 8 packed values (exact: the maximum of 16-bit floats is one of them).  The signs go with the comparison, not by eight masks
// before it: quantizer 4096 x 4096 9.2 -> 8.9 us, 16384 x 4096 28.0 -> 27.8.
template <typename T>
__device__ __forceinline__ float amax8(const uint4& raw) {
  const uint32_t w = Pk<T>::max2(Pk<T>::absmax2(raw.x, raw.y), Pk<T>::absmax2(raw.z, raw.w));
  return fmaxf(Pk<T>::lo(w), Pk<T>::hi(w));
}

// 32 bytes in one load
__device__ __forceinline__ void ldg_stream_v8(const void* p, uint4& a, uint4& b) {
  asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
               : "l"(p));
}

// Quantizes one block of 16 with the scale byte's exact arithmetic: codes and scale byte.  multiplier(sfb) is what the values are
// multiplied with before they are rounded to E2M1: out_scale_of(sfb, 1 / global scale), or a table of it.
template <typename T, typename Multiplier>
__device__ __forceinline__ uint2 quantize_block16(const uint4& r0, const uint4& r1, float gs, Multiplier&& multiplier, uint32_t& sfb) {
  const float amax = fmaxf(amax8<T>(r0), amax8<T>(r1));
  sfb = f32_to_e4m3(fminf(__fmul_rn(gs, __fmul_rn(amax, 0.16666667163372039794921875f)), 448.f));    // fl32(1/6)
  const float os = multiplier(sfb);
  float v[16];
  unpack8<T>(r0, v);
  unpack8<T>(r1, v + 8);
  return make_uint2(f32x8_to_e2m1(__fmul_rn(v[0], os), __fmul_rn(v[1], os), __fmul_rn(v[2], os), __fmul_rn(v[3], os),
                                  __fmul_rn(v[4], os), __fmul_rn(v[5], os), __fmul_rn(v[6], os), __fmul_rn(v[7], os)),
                    f32x8_to_e2m1(__fmul_rn(v[8], os), __fmul_rn(v[9], os), __fmul_rn(v[10], os), __fmul_rn(v[11], os),
                                  __fmul_rn(v[12], os), __fmul_rn(v[13], os), __fmul_rn(v[14], os), __fmul_rn(v[15], os)));
}

}  // namespace b200fp4
