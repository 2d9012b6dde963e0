// One MoE layer over dense NVFP4 expert weights in one call: routing metadata -> token-major quantization -> grouped
// gate_up GEMM with SiLU*up and quantization in its epilogue -> grouped down GEMM -> un-permute and weighted sum (the flow of
// vllm/model_executor/layers/fused_moe/experts/cutlass_moe.py:567-663).  Issued as separate Python calls a prompt of a few
// hundred tokens spent 130 us on the host for 200 us of kernels.
#include "common.cuh"

namespace b200fp4 {
namespace {

size_t part(size_t v) { return (v + 255) / 256 * 256; }

struct PrefillLayout {
  int64_t P, sf_rows;
  size_t eo, bso, dst2src, src2dst, xq, xsf, hq, hsf, c2, gemm, total;
};

PrefillLayout prefill_layout(int64_t M, int64_t topk, int64_t H, int64_t I, int64_t E) {
  PrefillLayout l;
  l.P = M * topk;
  l.sf_rows = (l.P + 127) / 128 * 128 + 128 * E;
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t here = at;
    at += part(bytes);
    return here;
  };
  l.eo = take((size_t)(E + 1) * 4);
  l.bso = take((size_t)(E + 1) * 4);
  l.dst2src = take((size_t)l.P * 4);
  l.src2dst = take((size_t)l.P * 4);
  l.xq = take((size_t)l.P * H / 2);
  l.xsf = take((size_t)l.sf_rows * ((H / 16 + 3) / 4 * 4));
  l.hq = take((size_t)l.P * I / 2);
  l.hsf = take((size_t)l.sf_rows * ((I / 16 + 3) / 4 * 4));
  l.c2 = take((size_t)l.P * H * 2);
  l.gemm = take(b200fp4_grouped_gemm_workspace_bytes(l.P, E));
  l.total = at;
  return l;
}

}  // namespace
}  // namespace b200fp4

using namespace b200fp4;

extern "C" size_t b200fp4_moe_prefill_workspace_bytes(int64_t M, int64_t topk, int64_t H, int64_t I, int64_t E) {
  if (M <= 0 || topk <= 0 || H <= 0 || I <= 0 || E <= 0) return 0;
  return prefill_layout(M, topk, H, I, E).total;
}

extern "C" int b200fp4_moe_prefill(const void* hidden, int dtype, const float* topk_weights, const int32_t* topk_ids,
                                   const int32_t* expert_map, int64_t global_E, const void* w13_codes, const void* w13_sf,
                                   const float* alpha1, const void* w2_codes, const void* w2_sf, const float* alpha2,
                                   const float* a1_gs, const float* a2_gs, void* out, int64_t M, int64_t topk, int64_t H, int64_t I,
                                   int64_t E, void* workspace, size_t workspace_bytes, void* stream) {
  if (M < 0 || topk <= 0 || topk > 32 || H <= 0 || H % 64 != 0 || I <= 0 || I % 128 != 0 || E <= 0) return B200FP4_STATUS_INVALID_VALUE;
  if (M == 0) return B200FP4_STATUS_SUCCESS;
  const PrefillLayout l = prefill_layout(M, topk, H, I, E);
  if (!workspace || !aligned(workspace, 256) || workspace_bytes < l.total) return B200FP4_STATUS_ALLOC_FAILED;
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  int32_t* eo = reinterpret_cast<int32_t*>(ws + l.eo);
  int32_t* bso = reinterpret_cast<int32_t*>(ws + l.bso);
  int32_t* dst2src = reinterpret_cast<int32_t*>(ws + l.dst2src);
  int32_t* src2dst = reinterpret_cast<int32_t*>(ws + l.src2dst);
  const size_t gemm_bytes = b200fp4_grouped_gemm_workspace_bytes(l.P, E);
  int rc = b200fp4_moe_permute(topk_ids, expert_map, global_E, M, topk, E, eo, bso, dst2src, src2dst, stream);
  if (rc == B200FP4_STATUS_SUCCESS)
    rc = b200fp4_experts_quantize_scatter(hidden, dtype, M, H, topk, src2dst, a1_gs, eo, bso, (int32_t)E, l.sf_rows, topk_ids, expert_map,
                                          global_E, ws + l.xq, ws + l.xsf, stream);
  if (rc == B200FP4_STATUS_SUCCESS)
    rc = b200fp4_grouped_gemm_nvfp4_silu_quant(ws + l.xq, w13_codes, ws + l.xsf, w13_sf, alpha1, eo, bso, a2_gs, dtype, ws + l.hq,
                                               ws + l.hsf, l.P, 2 * I, H, E, ws + l.gemm, gemm_bytes, stream);
  if (rc == B200FP4_STATUS_SUCCESS)
    rc = b200fp4_grouped_gemm_nvfp4(ws + l.hq, w2_codes, ws + l.hsf, w2_sf, alpha2, eo, bso, ws + l.c2, dtype, l.P, H, I, E, 0,
                                    ws + l.gemm, gemm_bytes, stream);
  if (rc == B200FP4_STATUS_SUCCESS)
    rc = b200fp4_moe_unpermute_reduce(ws + l.c2, dtype, src2dst, topk_weights, M, topk, H, out, stream);
  return rc;
}
