// The MoE decode layer's two projections for few (token, expert) pairs (moe_small.cu): which calls it takes, and its launch.
#pragma once

#include "sparse_mma.cuh"

namespace b200fp4 {

struct MoeSmallArgs {
  SparseWeights w13, w2;
  const void* hidden;               // [M, H] bf16 / f16, rows ld_h elements apart
  int64_t ld_h;
  const int32_t* ids;               // [M, topk], rows ids_ld apart
  int64_t ids_ld;
  const int32_t* expert_map;
  int global_E, E, topk, H, I;
  int* status;                      // status word of the layer: cleared
  float* down;                      // [P, H]: written, but for the rows of experts that are not local
};

// Blocks per pair, or 0 where the general path is to be taken.  Both projections in the layout of the warp-scheduled kernels, ordered metadata;
// local: how many of the P pairs are expected to have their expert here.
int moe_small_cluster(int64_t P, double local, int64_t H, int64_t I);
int launch_moe_small(int cluster, bool bf16, const MoeSmallArgs& a, int64_t P, cudaStream_t st);

}  // namespace b200fp4
