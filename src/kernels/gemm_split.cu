// bf16 GEMM for problems with too few 256-column tiles to occupy the chip: one tile of 128 rows x
// BNT columns (64, 128 or 256) per CTA, or per cluster of S CTAs that cut its K loop.
//
//   warp 0      : TMA producer
//   warp 1      : UMMA issuer (tcgen05.mma.cta_group::1, one accumulator of BNT TMEM columns)
//   warps 2..5  : epilogue
//
// S > 1: CTA r of the cluster multiplies the r-th part of the K range.  When all CTAs have their
// partial tile in TMEM, every CTA sends each 32 x 32 piece of it (float32) into the shared memory
// of the piece's owner, and the owner adds the S partials in rank order, in float32, and runs the
// epilogue once: no workspace, no second kernel, one rounding, the same bits in every run.  The
// exchange re-uses the operand ring (all MMAs of the cluster have retired by then).
//
// The grid is not persistent: a CTA handles one tile and two CTAs fit on an SM when the ring is
// kept small, so one CTA's epilogue runs beside the other's main loop.
#include <map>
#include <mutex>

#include "gemm_device.cuh"
#include "gemm_split.cuh"
#include "launch_count.h"

namespace mgk {
namespace gemm {

namespace {

constexpr int SPLIT_THREADS = 192;
constexpr int A_TILE_BYTES = BM * BK * 2;   // 16 KB
constexpr int PIECE_BYTES = 32 * 32 * 4;    // float32 partials of 32 rows x 32 columns
constexpr int MAX_STAGES = 8;
constexpr int EPI_STAGING = 4 * 2 * OUT_BOX_BYTES;  // two boxes per epilogue warp
constexpr int BAR_BYTES = 256;

constexpr int stage_bytes(int bnt) { return A_TILE_BYTES + bnt * BK * 2; }
// Smallest ring: with S > 1 it has to hold the exchanged partials (BNT x 128 float32) and the
// staging boxes, without only the staging boxes.  Two stages at least, which also keeps the sum of
// the TMEM columns of the CTAs that fit on one SM within 512: an allocation never waits for a
// CTA that in turn waits for a cluster peer.
constexpr int min_stages(int bnt, bool split) {
    const int need = split ? bnt * 512 + EPI_STAGING : EPI_STAGING;
    const int st = (need + stage_bytes(bnt) - 1) / stage_bytes(bnt);
    return st < 2 ? 2 : st;
}

struct SParams {
    int M, N, K;
    SplitRaster raster;
    int stages;
    const __nv_bfloat16* D;  // EPI_ACCUM reads it
    long ldd;
    const __nv_bfloat16* aux;
    long ldaux;
    int aux_off;
    const int* m_block_group;
    int group_rows_b;
    const int* k_begin;
    const int* k_end;
    int* error_flag;
    uint64_t wait_limit_ns;
};

__device__ __forceinline__ uint32_t cluster_nctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d)
                 : "memory");
}

// The epilogue of 32 rows x 32 columns: lane = row, `r` the accumulator (for SwiGLU the gate, with
// the up values in `ru`).  `row0` is the first of the 32 rows, `drow0` its row of D.
template <int EPI>
__device__ __forceinline__ void finish_piece(const SParams& p, uint32_t (&r)[32], uint32_t (&ru)[32], int row0,
                                             long drow0, int col, int lane, OutRing& out) {
    const int ok = p.N - col;
    if (row0 >= p.M || ok <= 0)
        return;
    const bool row_ok = row0 + lane < p.M;
    const long drow = drow0 + lane;
    const int box_row = static_cast<int>(drow0);
    uint32_t pk[16], pk2[16];
    if (EPI == EPI_SWIGLU) {
        uint32_t ph[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float g0 = __uint_as_float(r[2 * i]), g1 = __uint_as_float(r[2 * i + 1]);
            const float u0 = __uint_as_float(ru[2 * i]), u1 = __uint_as_float(ru[2 * i + 1]);
            pk[i] = pack_bf16x2(g0, g1);
            pk2[i] = pack_bf16x2(u0, u1);
            ph[i] = pack_bf16x2(__fdividef(g0, 1.f + __expf(-g0)) * u0, __fdividef(g1, 1.f + __expf(-g1)) * u1);
        }
        emit_box32(out.map_d, out, lane, col, box_row, pk);
        emit_box32(out.map_du, out, lane, col, box_row, pk2);
        emit_box32(out.map_d2, out, lane, col, box_row, ph);
    } else if (EPI == EPI_STORE_F32) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            pk[i] = r[i];
            pk2[i] = r[16 + i];
        }
        emit_box32(out.map_d, out, lane, col, box_row, pk);
        if (ok > 16)
            emit_box32(out.map_d, out, lane, col + 16, box_row, pk2);
    } else if (EPI == EPI_DSWIGLU) {
        uint32_t cg[16], cu[16];
        if (row_ok) {
            load_packed32(p.aux + drow * p.ldaux + col, cg, ok);
            load_packed32(p.aux + drow * p.ldaux + p.aux_off + col, cu, ok);
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i)
                cg[i] = cu[i] = 0u;
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float dgv[2], duv[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float g = h ? bf16_hi(cg[i]) : bf16_lo(cg[i]);
                const float u = h ? bf16_hi(cu[i]) : bf16_lo(cu[i]);
                const float sg = __fdividef(1.f, 1.f + __expf(-g));
                const float dh = __uint_as_float(r[2 * i + h]);
                const float silu = g * sg;
                dgv[h] = dh * u * (sg + silu * (1.f - sg));  // dG
                duv[h] = dh * silu;                           // dU
            }
            pk[i] = pack_bf16x2(dgv[0], dgv[1]);
            pk2[i] = pack_bf16x2(duv[0], duv[1]);
        }
        emit_box32(out.map_d, out, lane, col, box_row, pk);
        emit_box32(out.map_du, out, lane, col, box_row, pk2);
    } else {
        float o[32];
        if (EPI == EPI_ACCUM && row_ok) {
            load_row32(p.D + drow * p.ldd + col, o, ok);
        } else {
#pragma unroll
            for (int i = 0; i < 32; ++i)
                o[i] = 0.f;
        }
#pragma unroll
        for (int i = 0; i < 16; ++i)
            pk[i] = EPI == EPI_ACCUM ? pack_bf16x2(__uint_as_float(r[2 * i]) + o[2 * i],
                                                   __uint_as_float(r[2 * i + 1]) + o[2 * i + 1])
                                     : pack_bf16x2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
        emit_box32(out.map_d, out, lane, col, box_row, pk);
    }
}

template <int BNT, bool A_MN, bool B_MN, int EPI>
__global__ void __launch_bounds__(SPLIT_THREADS, 2)
        gemm_split_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                          const __grid_constant__ CUtensorMap tma_d, const __grid_constant__ CUtensorMap tma_du,
                          const __grid_constant__ CUtensorMap tma_d2, const SParams p) {
    constexpr int B_TILE_BYTES = BNT * BK * 2;
    constexpr int STAGE = A_TILE_BYTES + B_TILE_BYTES;
    constexpr int SETS = EPI == EPI_SWIGLU ? 2 : 1;   // accumulator pieces that one output piece needs
    constexpr int CHUNKS = BNT / 32 / SETS;           // 32-column output chunks of a tile
    constexpr int PIECES = CHUNKS * 4;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                               ~static_cast<uintptr_t>(1023));
    const int stages = p.stages;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + stages * STAGE);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * MAX_STAGES + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int lane = threadIdx.x & 31;
    const int splits = static_cast<int>(cluster_nctarank());
    const int crank = static_cast<int>(cluster_ctarank());

    const uint32_t full0 = smem_u32(bars);
    const uint32_t empty0 = smem_u32(bars + MAX_STAGES);
    const uint32_t tfull = smem_u32(bars + 2 * MAX_STAGES);

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        prefetch_tensormap(&tma_a);
        prefetch_tensormap(&tma_b);
        for (int s = 0; s < stages; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        mbar_init(tfull, 1);
        mbar_fence_init();
        fence_proxy_async_smem();
    }
    if (warp == 1) {
        tmem_alloc_cg1(smem_u32(tmem_slot), BNT);
        tmem_relinquish_cg1();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    // ---- this cluster's tile and this CTA's part of its K range
    int t = static_cast<int>(blockIdx.x) / splits;
    int grp = 0;
    if (p.k_begin != nullptr) {
        const int per = p.raster.m_blocks * p.raster.n_blocks;
        grp = t / per;
        t -= grp * per;
    }
    const SplitTile tile = split_tile(p.raster, t);
    const int mb = tile.m_block;
    const int m0 = mb * BM;
    const int n0 = tile.n_block * p.raster.n_tile_stride;
    long drow0 = m0;
    int b_row = 0, k_first = 0, k_blocks = (p.K + BK - 1) / BK;
    bool skip = false;
    if (p.k_begin != nullptr) {
        k_first = p.k_begin[grp];
        k_blocks = max(0, (p.k_end[grp] - k_first + BK - 1) / BK);
        drow0 = static_cast<long>(grp) * p.M + m0;
    } else if (p.m_block_group != nullptr) {
        const int e = p.m_block_group[mb];
        skip = e < 0;  // padding block: the whole cluster has nothing to do
        b_row = skip ? 0 : e * p.group_rows_b;
    }
    const int kb_begin = static_cast<int>(static_cast<long>(k_blocks) * crank / splits);
    const int kb_end = skip ? kb_begin : static_cast<int>(static_cast<long>(k_blocks) * (crank + 1) / splits);
    const bool has_acc = kb_end > kb_begin;

    WaitCtx wc{abort_flag, p.wait_limit_ns};

    // (both loops look at the next stage's barrier while this one's work is issued: a wait that is
    // already over costs 170 cycles if it is only then asked for)
    if (warp == 0) {
        if (elect_one()) {
            int s = 0;
            uint32_t ph = 0;
            bool ready = false;
            for (int kb = kb_begin; kb < kb_end; ++kb) {
                if (!ready && !mbar_wait(empty0 + 8 * s, ph ^ 1, wc))
                    break;
                const int k = k_first + kb * BK;
                const uint32_t sa = smem_u32(smem + s * STAGE), sb = sa + A_TILE_BYTES;
                const uint32_t fb = full0 + 8 * s;
                if (++s == stages) {
                    s = 0;
                    ph ^= 1;
                }
                ready = mbar_test_wait(empty0 + 8 * s, ph ^ 1);
                mbar_expect_tx(fb, STAGE);
                if (!A_MN) {
                    tma_load_2d(sa, &tma_a, fb, k, m0);
                } else {
#pragma unroll
                    for (int j = 0; j < BM / 64; ++j)
                        tma_load_2d(sa + j * MN_CHUNK_BYTES, &tma_a, fb, m0 + 64 * j, k);
                }
                if (EPI == EPI_SWIGLU) {
                    tma_load_2d(sb, &tma_b, fb, k, b_row + n0);
                    tma_load_2d(sb + B_TILE_BYTES / 2, &tma_b, fb, k, b_row + n0 + p.aux_off);
                } else if (!B_MN) {
                    tma_load_2d(sb, &tma_b, fb, k, b_row + n0);
                } else {
#pragma unroll
                    for (int j = 0; j < BNT / 64; ++j)
                        tma_load_2d(sb + j * MN_CHUNK_BYTES, &tma_b, fb, n0 + 64 * j, b_row + k);
                }
            }
        }
    } else if (warp == 1) {
        if (has_acc && elect_one()) {
            constexpr uint32_t idesc = umma_idesc_bf16_f32(BM, BNT, A_MN, B_MN);
            int s = 0;
            uint32_t ph = 0;
            bool alive = true, ready = false;
            for (int kb = kb_begin; kb < kb_end; ++kb) {
                if (!ready && !mbar_wait(full0 + 8 * s, ph, wc)) {
                    alive = false;
                    break;
                }
                tc_fence_after();
                const uint32_t sa = smem_u32(smem + s * STAGE), sb = sa + A_TILE_BYTES;
                const uint32_t freed = empty0 + 8 * s;
                if (++s == stages) {
                    s = 0;
                    ph ^= 1;
                }
                ready = mbar_test_wait(full0 + 8 * s, ph);
#pragma unroll
                for (int kk = 0; kk < BK / UMMA_K; ++kk) {
                    const uint64_t ad = A_MN ? umma_smem_desc_sw128(sa + kk * (UMMA_K * 128), MN_CHUNK_BYTES, 1024)
                                             : umma_smem_desc_sw128(sa + kk * (UMMA_K * 2), 16, 1024);
                    const uint64_t bd = B_MN ? umma_smem_desc_sw128(sb + kk * (UMMA_K * 128), MN_CHUNK_BYTES, 1024)
                                             : umma_smem_desc_sw128(sb + kk * (UMMA_K * 2), 16, 1024);
                    umma_f16_cg1(tmem_base, ad, bd, idesc, (kb > kb_begin || kk != 0) ? 1u : 0u);
                }
                umma_commit_cg1(freed);
            }
            if (alive)
                umma_commit_cg1(tfull);
        }
    }

    OutRing out;
    out.nslots = 2;
    out.slot = 0;
    out.map_d = &tma_d;
    out.map_du = &tma_du;
    out.map_d2 = &tma_d2;
    const int q = warp & 3;  // TMEM lane quarter of an epilogue warp
    bool got = true;
    if (warp >= 2 && has_acc) {
        got = lane == 0 ? mbar_wait(tfull, 0, wc) : true;
        got = __all_sync(0xffffffffu, got);
        tc_fence_after();
    }
    const uint32_t t_addr = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    auto load_acc = [&](int column, uint32_t(&r)[32]) {
        if (has_acc) {
            tmem_ld_32x32b_x32(t_addr + column, r);
        } else {
#pragma unroll
            for (int i = 0; i < 32; ++i)
                r[i] = 0u;
        }
    };

    if (splits == 1) {
        if (warp >= 2 && got && !skip) {
            out.base = smem + q * 2 * OUT_BOX_BYTES;  // the ring is idle: every MMA has retired
#pragma unroll 1
            for (int c = 0; c < CHUNKS; ++c) {
                uint32_t r[32], ru[32];
                load_acc(c * 32, r);
                if (SETS == 2)
                    load_acc(BNT / 2 + c * 32, ru);
                if (has_acc) {
                    tmem_ld_wait(r);
                    if (SETS == 2)
                        tmem_ld_wait(ru);
                }
                finish_piece<EPI>(p, r, ru, m0 + q * 32, drow0 + q * 32, n0 + c * 32, lane, out);
            }
            if (elect_one())
                tma_store_wait<0>();
        }
    } else {
        const int per_owner = PIECES / splits;
        __syncwarp();
        cluster_sync_all();  // every CTA of the cluster has finished its main loop: all rings are idle
        if (warp >= 2 && got && !skip) {
            // piece (chunk c, row quarter q) goes to slot [piece of the owner][this rank][set]; the
            // 16-byte vector j of lane l sits at j * 512 + l * 16: no bank conflicts on either side
#pragma unroll 1
            for (int c = 0; c < CHUNKS; ++c) {
                const int piece = c * 4 + q;
                const int owner = piece / per_owner;
                const uint32_t slot =
                        smem_u32(smem) + ((piece - owner * per_owner) * splits + crank) * (SETS * PIECE_BYTES) + lane * 16;
                const uint32_t dst = mapa_u32(slot, static_cast<uint32_t>(owner));
                uint32_t r[32], ru[32];
                load_acc(c * 32, r);
                if (SETS == 2)
                    load_acc(BNT / 2 + c * 32, ru);
                if (has_acc) {
                    tmem_ld_wait(r);
                    if (SETS == 2)
                        tmem_ld_wait(ru);
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    st_cluster_v4(dst + j * 512, r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
                    if (SETS == 2)
                        st_cluster_v4(dst + PIECE_BYTES + j * 512, ru[4 * j], ru[4 * j + 1], ru[4 * j + 2], ru[4 * j + 3]);
                }
            }
        }
        __syncwarp();
        cluster_sync_all();  // all partials have arrived
        if (warp >= 2 && got && !skip) {
            out.base = smem + BNT * 512 + q * 2 * OUT_BOX_BYTES;
#pragma unroll 1
            for (int i = warp - 2; i < per_owner; i += 4) {
                const int piece = crank * per_owner + i;
                const int c = piece >> 2, pq = piece & 3;
                const uint8_t* src = smem + i * splits * (SETS * PIECE_BYTES) + lane * 16;
                float acc[SETS][32];
#pragma unroll
                for (int set = 0; set < SETS; ++set)
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        acc[set][j] = 0.f;
#pragma unroll 1
                for (int rk = 0; rk < splits; ++rk) {
#pragma unroll
                    for (int set = 0; set < SETS; ++set) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const float4 v = *reinterpret_cast<const float4*>(src + (rk * SETS + set) * PIECE_BYTES + j * 512);
                            acc[set][4 * j] += v.x;
                            acc[set][4 * j + 1] += v.y;
                            acc[set][4 * j + 2] += v.z;
                            acc[set][4 * j + 3] += v.w;
                        }
                    }
                }
                uint32_t r[32], ru[32];
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    r[j] = __float_as_uint(acc[0][j]);
                    ru[j] = __float_as_uint(acc[SETS - 1][j]);
                }
                finish_piece<EPI>(p, r, ru, m0 + pq * 32, drow0 + pq * 32, n0 + c * 32, lane, out);
            }
            if (elect_one())
                tma_store_wait<0>();
        }
    }
    // ---------------------------------------------------------- teardown
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        // a wait ran out: loads already issued land within microseconds; shared memory is kept until then
        const uint64_t begin = globaltimer_ns();
        while (globaltimer_ns() - begin < 200000) {
        }
        if (threadIdx.x == 0 && p.error_flag != nullptr)
            atomicExch(p.error_flag, 1);
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_cg1(tmem_base, BNT);
    }
}

template <int BNT, bool A_MN, bool B_MN, int EPI>
cudaError_t launch_t(const Maps& maps, const SParams& sp, int splits, int tiles, cudaStream_t stream) {
    auto kern = gemm_split_kernel<BNT, A_MN, B_MN, EPI>;
    const int smem = sp.stages * stage_bytes(BNT) + 1024 /*align slack*/ + BAR_BYTES;
    int dev = 0;
    cudaGetDevice(&dev);
    {
        static std::mutex mu;
        static std::map<int, bool> ready;  // per device: the shared-memory attribute is set
        std::lock_guard<std::mutex> lk(mu);
        if (!ready[dev]) {
            const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
            if (e != cudaSuccess)
                return e;
            ready[dev] = true;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(tiles * splits));
    cfg.blockDim = dim3(SPLIT_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attrs[1];
    attrs[0].id = cudaLaunchAttributeClusterDimension;
    attrs[0].val.clusterDim.x = static_cast<unsigned>(splits);
    attrs[0].val.clusterDim.y = 1;
    attrs[0].val.clusterDim.z = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, maps.a, maps.b, maps.d, maps.du, maps.d2, sp);
    count_launch();
    return e;
}

template <int BNT, bool A_MN, bool B_MN>
cudaError_t launch_e(int epi, const Maps& m, const SParams& sp, int splits, int tiles, cudaStream_t stream) {
    switch (epi) {
        case EPI_STORE:
            return launch_t<BNT, A_MN, B_MN, EPI_STORE>(m, sp, splits, tiles, stream);
        case EPI_ACCUM:
            return launch_t<BNT, A_MN, B_MN, EPI_ACCUM>(m, sp, splits, tiles, stream);
        case EPI_STORE_F32:
            return launch_t<BNT, A_MN, B_MN, EPI_STORE_F32>(m, sp, splits, tiles, stream);
        case EPI_DSWIGLU:
            return launch_t<BNT, A_MN, B_MN, EPI_DSWIGLU>(m, sp, splits, tiles, stream);
        case EPI_SWIGLU:
            if (B_MN)
                return cudaErrorInvalidValue;
            return launch_t<BNT, A_MN, false, EPI_SWIGLU>(m, sp, splits, tiles, stream);
        default:
            return cudaErrorInvalidValue;
    }
}

template <int BNT>
cudaError_t launch_l(bool a_mn, bool b_mn, int epi, const Maps& m, const SParams& sp, int splits, int tiles,
                     cudaStream_t stream) {
    if (!a_mn && !b_mn)
        return launch_e<BNT, false, false>(epi, m, sp, splits, tiles, stream);
    if (!a_mn && b_mn)
        return launch_e<BNT, false, true>(epi, m, sp, splits, tiles, stream);
    if (a_mn && !b_mn)
        return launch_e<BNT, true, false>(epi, m, sp, splits, tiles, stream);
    return launch_e<BNT, true, true>(epi, m, sp, splits, tiles, stream);
}

}  // namespace

bool split_accepts(const GemmArgs& a, const SplitPlan& plan) {
    const bool grouped_k = a.grouped.k_begin != nullptr;
    if (a.epilogue != EPI_STORE && a.epilogue != EPI_ACCUM && a.epilogue != EPI_STORE_F32 &&
        a.epilogue != EPI_SWIGLU && a.epilogue != EPI_DSWIGLU)
        return false;
    if (a.epilogue == EPI_SWIGLU && a.b_mn)
        return false;
    if (a.a_ready != nullptr || a.fuse.ag_dst != nullptr || a.fuse.rs_out != nullptr || a.sm_limit > 0 || a.m_rot != 0)
        return false;
    if (grouped_k && a.M % BM)  // rows of a tile past M would land in the next group's result
        return false;
    if (plan.bn != 64 && plan.bn != 128 && plan.bn != 256)
        return false;
    const int pieces = plan.bn / 8 / (a.epilogue == EPI_SWIGLU ? 2 : 1);
    return (plan.splits == 1 || plan.splits == 2 || plan.splits == 4 || plan.splits == 8) && plan.splits <= pieces;
}

cudaError_t launch_gemm_split(const GemmArgs& a, const SplitPlan& plan, int sms, cudaStream_t stream) {
    if (!split_accepts(a, plan))
        return cudaErrorInvalidValue;
    const bool grouped_m = a.grouped.m_block_group != nullptr, grouped_k = a.grouped.k_begin != nullptr;
    const uint64_t groups = (grouped_m || grouped_k) ? static_cast<uint64_t>(a.grouped.groups) : 1;
    const bool swiglu = a.epilogue == EPI_SWIGLU;
    if ((swiglu || a.epilogue == EPI_DSWIGLU) && a.aux_off % 8)
        return cudaErrorInvalidValue;
    SParams sp{};
    sp.M = a.M;
    sp.N = a.N;
    sp.K = a.K;
    sp.raster = split_raster(a, plan);
    sp.D = static_cast<const __nv_bfloat16*>(a.D);
    sp.ldd = a.ldd;
    sp.aux = static_cast<const __nv_bfloat16*>(a.aux);
    sp.ldaux = a.ldaux;
    sp.aux_off = a.aux_off;
    sp.m_block_group = a.grouped.m_block_group;
    sp.group_rows_b = a.grouped.group_rows_b;
    sp.k_begin = a.grouped.k_begin;
    sp.k_end = a.grouped.k_end;
    sp.error_flag = a.error_flag;
    sp.wait_limit_ns = a.wait_limit_ns ? a.wait_limit_ns : 4000000000ull;
    const int tiles = sp.raster.m_blocks * sp.raster.n_blocks * (grouped_k ? static_cast<int>(groups) : 1);
    // Ring depth: all of shared memory when every CTA can have an SM of its own, half of it (two
    // CTAs per SM) otherwise; never more stages than the CTA has k-steps.
    const int kb = ((a.K + BK - 1) / BK + plan.splits - 1) / plan.splits;
    const int budget = (tiles * plan.splits <= sms ? 226 : 113) * 1024 - 1024 - BAR_BYTES;
    int stages = budget / stage_bytes(plan.bn);
    if (stages > kb)
        stages = kb;
    if (stages > MAX_STAGES)
        stages = MAX_STAGES;
    const int least = min_stages(plan.bn, plan.splits > 1);
    sp.stages = stages < least ? least : stages;

    Maps maps;
    bool ok = a.a_mn ? make_map(&maps.a, a.A, a.M, a.K, a.lda, BK) : make_map(&maps.a, a.A, a.K, a.M, a.lda, BM);
    if (!a.b_mn) {
        uint64_t rows = swiglu ? static_cast<uint64_t>(a.aux_off) + a.N : static_cast<uint64_t>(a.N);
        if (grouped_m)
            rows = groups * static_cast<uint64_t>(a.grouped.group_rows_b);
        ok = ok && make_map(&maps.b, a.B, a.K, rows, a.ldb, swiglu ? plan.bn / 2 : plan.bn);
    } else {
        const uint64_t krows = grouped_m ? groups * static_cast<uint64_t>(a.grouped.group_rows_b) : static_cast<uint64_t>(a.K);
        ok = ok && make_map(&maps.b, a.B, a.N, krows, a.ldb, BK);
    }
    const uint64_t out_rows = static_cast<uint64_t>(a.M) * (grouped_k ? groups : 1);
    ok = ok && make_out_map(&maps.d, a.D, a.N, out_rows, a.ldd, a.epilogue == EPI_STORE_F32);
    maps.du = maps.d2 = maps.d;
    if (ok && (swiglu || a.epilogue == EPI_DSWIGLU))
        ok = make_out_map(&maps.du, static_cast<const __nv_bfloat16*>(a.D) + a.aux_off, a.N, out_rows, a.ldd);
    if (ok && swiglu)
        ok = make_out_map(&maps.d2, a.D2, a.N, out_rows, a.ldd2);
    if (!ok)
        return cudaErrorInvalidValue;
    switch (plan.bn) {
        case 64:
            return launch_l<64>(a.a_mn, a.b_mn, a.epilogue, maps, sp, plan.splits, tiles, stream);
        case 128:
            return launch_l<128>(a.a_mn, a.b_mn, a.epilogue, maps, sp, plan.splits, tiles, stream);
        default:
            return launch_l<256>(a.a_mn, a.b_mn, a.epilogue, maps, sp, plan.splits, tiles, stream);
    }
}

}  // namespace gemm
}  // namespace mgk
