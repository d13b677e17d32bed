// Host side of the small-tile / cluster split-K GEMM kernel (gemm_split.cu).
#pragma once
#include "gemm_tcgen05.cuh"

namespace mgk {
namespace gemm {

struct SplitPlan {
    int bn;      // accumulator columns of a tile: 64, 128 or 256; 0 = do not use this kernel
    int splits;  // CTAs (a cluster) that share the K loop of one tile: 1, 2, 4 or 8
};

// Whether the kernel can run this problem with this plan.
bool split_accepts(const GemmArgs& a, const SplitPlan& plan);

// Launches it (operands already validated by launch_gemm_bf16).
cudaError_t launch_gemm_split(const GemmArgs& a, const SplitPlan& plan, int sms, cudaStream_t stream);

}  // namespace gemm
}  // namespace mgk
