// The GEMM of few tokens (gemm_small.cu): which calls it takes, and its launch.
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace b200fp4 {

constexpr int64_t kSmallMaxM = 64;

struct SmallPlan {
  bool ok;                // false: the general kernel's case
  int split, ring, stages, m_pad;
  size_t smem;
};
enum class SmallUse { kLinear, kLinearInGraph, kCodes, kCodesInGraph };      // quantizes its operand, given codes; launched, captured
SmallPlan small_gemm_plan(int64_t M, int64_t N, int64_t K, SmallUse use);

// gs given: x is [M, K] bf16 / f16 (rows ldx elements apart), quantized in the kernel; gs null: x are packed codes [M, K/2] and x_sf
// their swizzled scales.  mw: the weight [N, K/2] in boxes of 128 rows x 128 bytes.
int launch_gemm_small(const SmallPlan& plan, const CUtensorMap& mw, const void* x, int x_dtype, int64_t ldx, const float* gs, const uint8_t* x_sf,
                      const uint8_t* w_sf, const float* alpha, void* out, int out_dtype, int M, int N, int K, int* status, cudaStream_t st);

}  // namespace b200fp4
