// Host side of the small-tile / cluster split-K GEMM kernel (gemm_split.cu).
#pragma once
#include "gemm_tcgen05.cuh"

namespace mgk {
namespace gemm {

struct SplitPlan {
    int bn;      // accumulator columns of a tile: 64, 128 or 256; 0 = do not use this kernel
    int splits;  // CTAs (a cluster) that share the K loop of one tile: 1, 2, 4 or 8
};

// Output tiles of a problem (of each group, when the K ranges are grouped) and their order: sweeps of
// `group_m` row blocks over all columns, so that what runs together shares its operands in L2.
struct SplitRaster {
    int m_blocks, n_blocks;
    int group_m;
    int n_tile_stride;  // output columns of a tile: bn, or bn / 2 for the SwiGLU pairing
};
inline SplitRaster split_raster(const GemmArgs& a, const SplitPlan& plan) {
    const int cols = a.epilogue == EPI_SWIGLU ? plan.bn / 2 : plan.bn;
    return SplitRaster{(a.M + 127) / 128, (a.N + cols - 1) / cols, 16, cols};
}
struct SplitTile {
    int m_block, n_block;
};
__host__ __device__ __forceinline__ SplitTile split_tile(const SplitRaster& r, int t) {
    const int per_group = r.group_m * r.n_blocks;
    const int g = t / per_group;
    const int first_m = g * r.group_m;
    const int left = r.m_blocks - first_m;
    const int gsz = left < r.group_m ? left : r.group_m;
    return SplitTile{first_m + (t - g * per_group) % gsz, (t - g * per_group) / gsz};
}

// Whether the kernel can run this problem with this plan.
bool split_accepts(const GemmArgs& a, const SplitPlan& plan);

// Launches it (operands already validated by launch_gemm_bf16).
cudaError_t launch_gemm_split(const GemmArgs& a, const SplitPlan& plan, int sms, cudaStream_t stream);

}  // namespace gemm
}  // namespace mgk
