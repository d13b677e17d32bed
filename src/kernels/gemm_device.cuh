// Device and host pieces shared by the bf16 GEMM kernels: bf16 row access, cluster helpers, the
// staging ring of the TMA-store epilogues and the tensor maps.
#pragma once
#include "gemm_tcgen05.cuh"

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <mutex>

#include "ptx_sm100.cuh"

namespace mgk {
namespace gemm {

using namespace mgk::ptx;

namespace {

constexpr int BM = 128;  // rows of A per CTA
constexpr int BN = 256;  // accumulator columns
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int MN_CHUNK_BYTES = 64 * BK * 2;  // one 64(mn) x 64(k) box of an MN-major operand

__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

// 32 consecutive bf16 of one row as 16 packed words; columns from `ncols_ok` on read as zero
__device__ __forceinline__ void load_packed32(const __nv_bfloat16* src, uint32_t (&w)[16], int ncols_ok) {
    if (ncols_ok >= 32) {
        const uint4* s4 = reinterpret_cast<const uint4*>(src);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint4 q = s4[i];
            w[4 * i] = q.x; w[4 * i + 1] = q.y; w[4 * i + 2] = q.z; w[4 * i + 3] = q.w;
        }
    } else {
        const uint16_t* s16 = reinterpret_cast<const uint16_t*>(src);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const uint32_t lo16 = 2 * i < ncols_ok ? s16[2 * i] : 0u;
            const uint32_t hi16 = 2 * i + 1 < ncols_ok ? s16[2 * i + 1] : 0u;
            w[i] = lo16 | (hi16 << 16);
        }
    }
}
__device__ __forceinline__ void load_row32(const __nv_bfloat16* src, float (&v)[32], int ncols_ok) {
    if (ncols_ok >= 32) {
        const uint4* s4 = reinterpret_cast<const uint4*>(src);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint4 o = s4[i];
            v[i * 8 + 0] = bf16_lo(o.x);
            v[i * 8 + 1] = bf16_hi(o.x);
            v[i * 8 + 2] = bf16_lo(o.y);
            v[i * 8 + 3] = bf16_hi(o.y);
            v[i * 8 + 4] = bf16_lo(o.z);
            v[i * 8 + 5] = bf16_hi(o.z);
            v[i * 8 + 6] = bf16_lo(o.w);
            v[i * 8 + 7] = bf16_hi(o.w);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 32; ++i)
            v[i] = (i < ncols_ok) ? __bfloat162float(src[i]) : 0.f;
    }
}


// ---------------------------------------------------------------- cluster helpers
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of `addr` (a shared::cta address) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// TMA load issued by one CTA of a pair; its bytes complete on `bar` (a shared::cluster
// address, here the leader CTA's barrier).
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const void* map, uint32_t bar, int c0,
                                                 int c1) {
    asm volatile(
            "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
            " [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
            "l"(map), "r"(bar), "r"(c0), "r"(c1)
            : "memory");
}
// Completes the barrier at `bar` in both CTAs of the pair when all prior MMAs of this thread retire.
__device__ __forceinline__ void umma_commit_both(uint32_t bar) {
    asm volatile(
            "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                    bar),
            "h"(static_cast<uint16_t>(3))
            : "memory");
}
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr)
                 : "memory");
}

// One epilogue warp's way out to global memory for the TMA-store epilogues: a ring of 2 KB
// staging boxes (32 rows x 32 bf16, 64-byte swizzle) and the output tensor maps.  One elected lane
// issues every store of the warp, so its bulk groups count them.
struct OutRing {
    uint8_t* base;
    int nslots;  // 2 or 4
    int slot;
    const CUtensorMap* map_d;   // D, columns [0, N)
    const CUtensorMap* map_du;  // D + aux_off, columns [0, N): the second half of a gate/up pair
    const CUtensorMap* map_d2;  // D2
};
constexpr int OUT_BOX_BYTES = 32 * 32 * 2;

// Stores the warp's 32 rows x 32 columns (lane = row, 16 packed pairs) at (row, col) of `map`;
// the tensor map clips what lies past the matrix.
__device__ __forceinline__ void emit_box32(const CUtensorMap* map, OutRing& ring, int lane, int col, int row,
                                           const uint32_t (&pk)[16]) {
    // the store that last used this box has read it
    if (elect_one()) {
        if (ring.nslots == 2)
            tma_store_wait_read<1>();
        else
            tma_store_wait_read<3>();
    }
    __syncwarp();
    uint8_t* buf = ring.base + ring.slot * OUT_BOX_BYTES;
    const int sw = (lane >> 1) & 3;  // 64-byte swizzle: 16-byte piece index ^ address bits 7..8
#pragma unroll
    for (int j = 0; j < 4; ++j)
        *reinterpret_cast<uint4*>(buf + lane * 64 + ((j ^ sw) << 4)) =
                make_uint4(pk[4 * j], pk[4 * j + 1], pk[4 * j + 2], pk[4 * j + 3]);
    fence_proxy_async_smem();
    __syncwarp();
    if (elect_one()) {
        tma_store_2d(map, smem_u32(buf), col, row);
        tma_store_commit();
    }
    ring.slot = ring.slot + 1 == ring.nslots ? 0 : ring.slot + 1;
}

// ------------------------------------------------------------------ host side

PFN_cuTensorMapEncodeTiled_v12000 get_encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) ==
                    cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
    });
    return fn;
}

// bf16 matrix, `inner` contiguous elements per row, `outer` rows `ld` elements apart;
// box = 64 inner elements (128 B, the swizzle span) x `box_rows`.
bool make_map(CUtensorMap* map, const void* ptr, uint64_t inner, uint64_t outer, uint64_t ld,
              uint32_t box_rows) {
    auto fn = get_encode_fn();
    if (fn == nullptr)
        return false;
    cuuint64_t dims[2] = {inner, outer};
    cuuint64_t strides[1] = {ld * 2};
    cuuint32_t box[2] = {64, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides,
                    box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

// Output matrix for the TMA-store epilogues: box = 32 columns (64 B, the swizzle span) x 32 rows;
// for a float32 matrix 16 columns x 32 rows (the same 64-byte rows).
bool make_out_map(CUtensorMap* map, const void* ptr, uint64_t cols, uint64_t rows, uint64_t ld, bool f32 = false) {
    auto fn = get_encode_fn();
    if (fn == nullptr)
        return false;
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {ld * (f32 ? 4u : 2u)};
    cuuint32_t box[2] = {f32 ? 16u : 32u, 32};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides,
                    box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                    CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

struct Maps {
    CUtensorMap a, b, d, du, d2;
};

}  // namespace
}  // namespace gemm
}  // namespace mgk
