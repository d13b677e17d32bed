#include "elementwise.cuh"

#include <cuda_bf16.h>

#include "launch_count.h"

namespace mgk {
namespace ew {

namespace {

__device__ __forceinline__ float lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
__device__ __forceinline__ uint32_t pack(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
}

// 32 consecutive bytes of global memory: one 256-bit access when the address allows it, else two
// of 128 bits.  Data that is used once does not displace anything in L1.
template <bool WIDE>
__device__ __forceinline__ void load32(const void* p, uint32_t (&r)[8]) {
    if (WIDE) {
        asm volatile("ld.global.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "l"(p));
    } else {
        const uint4 a = __ldcs(static_cast<const uint4*>(p)), b = __ldcs(static_cast<const uint4*>(p) + 1);
        r[0] = a.x; r[1] = a.y; r[2] = a.z; r[3] = a.w;
        r[4] = b.x; r[5] = b.y; r[6] = b.z; r[7] = b.w;
    }
}
template <bool WIDE>
__device__ __forceinline__ void store32(void* p, const uint32_t (&r)[8]) {
    if (WIDE) {
        asm volatile("st.global.v8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};" ::"r"(r[0]), "r"(r[1]), "r"(r[2]),
                     "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "l"(p)
                     : "memory");
    } else {
        static_cast<uint4*>(p)[0] = make_uint4(r[0], r[1], r[2], r[3]);
        static_cast<uint4*>(p)[1] = make_uint4(r[4], r[5], r[6], r[7]);
    }
}

// Bound by HBM: 14 bytes per element with a momentum buffer, 6 without.  A thread handles groups of
// 16 elements (32 bytes of weights and of gradients, 64 of momentum), all loads before the first
// use; the grid covers the bucket once, so that no wave of a grid-stride loop is left part empty.
// 25.6 M elements with momentum: 62.4 us in a grid-stride loop of 8 elements with 128-bit accesses,
// 55.5 us so (6.45 TB/s; a copy reaches 6.55).
template <bool MOM, bool WIDE>
__global__ void __launch_bounds__(256) sgd_bf16_kernel(__nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ g,
                                                       float* __restrict__ mom, uint64_t n, float lr, float mu, float wd) {
    constexpr int U = MOM ? 1 : 2;  // groups per thread
    const uint64_t groups = n / 16;
    const uint64_t first = static_cast<uint64_t>(blockIdx.x) * (256 * U) + threadIdx.x;
    uint32_t wv[U][8], gv[U][8], mv[U][2][8];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const uint64_t i = first + u * 256;
        if (i < groups) {
            load32<WIDE>(w + i * 16, wv[u]);
            load32<WIDE>(g + i * 16, gv[u]);
            if (MOM) {
                load32<WIDE>(mom + i * 16, mv[u][0]);
                load32<WIDE>(mom + i * 16 + 8, mv[u][1]);
            }
        }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const uint64_t i = first + u * 256;
        if (i >= groups)
            break;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            float wf[2] = {lo(wv[u][k]), hi(wv[u][k])};
            const float gf[2] = {lo(gv[u][k]), hi(gv[u][k])};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (MOM) {
                    uint32_t& slot = mv[u][k >> 2][(2 * k + h) & 7];
                    const float m = mu * __uint_as_float(slot) + gf[h] + wd * wf[h];
                    slot = __float_as_uint(m);
                    wf[h] -= lr * m;
                } else {
                    wf[h] -= lr * (gf[h] + wd * wf[h]);
                }
            }
            wv[u][k] = pack(wf[0], wf[1]);
        }
        store32<WIDE>(w + i * 16, wv[u]);
        if (MOM) {
            store32<WIDE>(mom + i * 16, mv[u][0]);
            store32<WIDE>(mom + i * 16 + 8, mv[u][1]);
        }
    }
    const uint64_t t = groups * 16 + threadIdx.x;  // fewer than 16 elements are left
    if (blockIdx.x == 0 && t < n) {
        float wf = __bfloat162float(w[t]);
        float gf = __bfloat162float(g[t]) + wd * wf;
        if (MOM) {
            mom[t] = mu * mom[t] + gf;
            gf = mom[t];
        }
        w[t] = __float2bfloat16_rn(wf - lr * gf);
    }
}

__global__ void __launch_bounds__(256) mse_bf16_kernel(const __nv_bfloat16* __restrict__ y,
                                                       const __nv_bfloat16* __restrict__ t,
                                                       __nv_bfloat16* __restrict__ dy, float* loss, uint64_t n,
                                                       float scale, int vec_ok) {
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    const uint64_t tid = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    float acc = 0.f;
    // 16-byte body (two vectors in flight per thread), scalar tail
    const uint64_t nvec = vec_ok ? n / 8 : 0;
    const uint4* yv = reinterpret_cast<const uint4*>(y);
    const uint4* tv = reinterpret_cast<const uint4*>(t);
    uint4* dv = reinterpret_cast<uint4*>(dy);
    auto one = [&](const uint4& a, const uint4& b, uint64_t i) {
        const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
        const uint32_t bw[4] = {b.x, b.y, b.z, b.w};
        uint32_t ow[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float d0 = lo(aw[k]) - lo(bw[k]);
            const float d1 = hi(aw[k]) - hi(bw[k]);
            acc += d0 * d0 + d1 * d1;
            ow[k] = pack(2.f * d0 * scale, 2.f * d1 * scale);
        }
        if (dy != nullptr)
            dv[i] = make_uint4(ow[0], ow[1], ow[2], ow[3]);
    };
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    // four independent vectors per thread and iteration, all loads issued before the first use
    constexpr int U = 4;
    uint64_t i = tid;
    for (; i + (U - 1) * stride < nvec; i += U * stride) {
        uint4 av[U], bv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            av[u] = __ldcs(yv + i + u * stride);
            bv[u] = t != nullptr ? __ldcs(tv + i + u * stride) : zero;
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            one(av[u], bv[u], i + u * stride);
    }
    for (; i < nvec; i += stride)
        one(__ldcs(yv + i), t != nullptr ? __ldcs(tv + i) : zero, i);
    for (uint64_t k = nvec * 8 + tid; k < n; k += stride) {
        const float d = __bfloat162float(y[k]) - (t != nullptr ? __bfloat162float(t[k]) : 0.f);
        acc += d * d;
        if (dy != nullptr)
            dy[k] = __float2bfloat16_rn(2.f * d * scale);
    }
    for (int o = 16; o > 0; o >>= 1)
        acc += __shfl_xor_sync(0xffffffffu, acc, o);
    __shared__ float part[8];
    if ((threadIdx.x & 31) == 0)
        part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        float s = 0.f;
        for (int k = 0; k < 8; ++k)
            s += part[k];
        atomicAdd(loss, s * scale);
    }
}


// One CTA of 256 threads per row; each thread keeps its 8-element vectors in registers so
// the row is read once.
constexpr int kNormThreads = 256;
constexpr int kNormMaxVec = 8;  // 256 threads * 8 vectors * 8 elements = 16384 columns

__device__ __forceinline__ float block_sum(float v, float* smem) {
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0)
        smem[threadIdx.x >> 5] = v;
    __syncthreads();
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < kNormThreads / 32; ++k)
        s += smem[k];
    __syncthreads();
    return s;
}

__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
    f[0] = lo(v.x); f[1] = hi(v.x); f[2] = lo(v.y); f[3] = hi(v.y);
    f[4] = lo(v.z); f[5] = hi(v.z); f[6] = lo(v.w); f[7] = hi(v.w);
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
    uint4 v;
    v.x = pack(f[0], f[1]); v.y = pack(f[2], f[3]); v.z = pack(f[4], f[5]); v.w = pack(f[6], f[7]);
    return v;
}

// NV = 16-byte vectors per thread; the row stays in registers as packed bf16 (4 registers per
// vector), which keeps several CTAs resident per SM.
template <int NV>
__global__ void __launch_bounds__(kNormThreads, NV <= 4 ? 4 : 2)
        add_rmsnorm_kernel(const uint4* __restrict__ x, const uint4* __restrict__ y, uint4* __restrict__ x_out,
                           uint4* __restrict__ n_out, float* __restrict__ inv_rms, int cols, float eps) {
    __shared__ float red[kNormThreads / 32];
    const int nvec = cols / 8;
    const size_t row = blockIdx.x;
    const uint4* xr = x + row * nvec;
    const uint4* yr = y != nullptr ? y + row * nvec : nullptr;
    uint4 xs[NV], ys[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        const int i = threadIdx.x + v * kNormThreads;
        if (i < nvec) {
            xs[v] = xr[i];
            if (yr != nullptr)
                ys[v] = __ldcs(yr + i);
        }
    }
    float ss = 0.f;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        const int i = threadIdx.x + v * kNormThreads;
        if (i < nvec) {
            float s[8];
            unpack8(xs[v], s);
            if (yr != nullptr) {
                float t[8];
                unpack8(ys[v], t);
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    s[k] += t[k];
                // the sum is rounded to bf16 where it is stored; normalise what was stored
                xs[v] = pack8(s);
                unpack8(xs[v], s);
            }
            if (x_out != nullptr)
                x_out[row * nvec + i] = xs[v];
#pragma unroll
            for (int k = 0; k < 8; ++k)
                ss += s[k] * s[k];
        }
    }
    if (n_out == nullptr && inv_rms == nullptr)
        return;
    const float total = block_sum(ss, red);
    const float r = rsqrtf(total / static_cast<float>(cols) + eps);
    if (inv_rms != nullptr && threadIdx.x == 0)
        inv_rms[row] = r;
    if (n_out != nullptr) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const int i = threadIdx.x + v * kNormThreads;
            if (i < nvec) {
                float o[8];
                unpack8(xs[v], o);
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    o[k] *= r;
                n_out[row * nvec + i] = pack8(o);
            }
        }
    }
}

template <int NV>
__global__ void __launch_bounds__(kNormThreads, NV <= 4 ? 4 : 2)
        rmsnorm_bwd_kernel(const uint4* __restrict__ dn, const uint4* __restrict__ n, const float* __restrict__ inv_rms,
                           const uint4* __restrict__ dres, uint4* __restrict__ dx, int cols) {
    __shared__ float red[kNormThreads / 32];
    const int nvec = cols / 8;
    const size_t row = blockIdx.x;
    uint4 gs[NV], ns[NV], ds[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        const int i = threadIdx.x + v * kNormThreads;
        if (i < nvec) {
            gs[v] = __ldcs(dn + row * nvec + i);
            ns[v] = __ldcs(n + row * nvec + i);
            if (dres != nullptr)
                ds[v] = __ldcs(dres + row * nvec + i);
        }
    }
    float dot = 0.f;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        const int i = threadIdx.x + v * kNormThreads;
        if (i < nvec) {
            float g[8], nn[8];
            unpack8(gs[v], g);
            unpack8(ns[v], nn);
#pragma unroll
            for (int k = 0; k < 8; ++k)
                dot += g[k] * nn[k];
        }
    }
    const float mean = block_sum(dot, red) / static_cast<float>(cols);
    const float r = inv_rms[row];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        const int i = threadIdx.x + v * kNormThreads;
        if (i < nvec) {
            float g[8], nn[8], o[8];
            unpack8(gs[v], g);
            unpack8(ns[v], nn);
#pragma unroll
            for (int k = 0; k < 8; ++k)
                o[k] = r * (g[k] - nn[k] * mean);
            if (dres != nullptr) {
                float d[8];
                unpack8(ds[v], d);
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    o[k] += d[k];
            }
            dx[row * nvec + i] = pack8(o);
        }
    }
}

// Smallest vectors-per-thread count that covers the row.
inline int norm_nv(int cols) {
    const int need = (cols / 8 + kNormThreads - 1) / kNormThreads;
    return need <= 1 ? 1 : need <= 2 ? 2 : need <= 4 ? 4 : 8;
}

}  // namespace

cudaError_t launch_sgd_bf16(void* w, const void* g, float* momentum, uint64_t n, float lr, float mu,
                            float weight_decay, cudaStream_t stream) {
    if (n == 0)
        return cudaSuccess;
    if ((reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(g)) & 15)
        return cudaErrorInvalidValue;
    // whole groups read and write the momentum in vectors, fewer than 16 elements one by one
    if (reinterpret_cast<uintptr_t>(momentum) & (n >= 16 ? 15 : 3))
        return cudaErrorInvalidValue;
    auto* wb = static_cast<__nv_bfloat16*>(w);
    auto* gb = static_cast<const __nv_bfloat16*>(g);
    const bool wide = ((reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(g) |
                        reinterpret_cast<uintptr_t>(momentum)) & 31) == 0;
    const uint64_t per_block = 256ull * 16 * (momentum != nullptr ? 1 : 2);
    const uint64_t blocks = (n + per_block - 1) / per_block;
    if (blocks > 0x7fffffffull)
        return cudaErrorInvalidValue;
    auto go = [&](auto kernel) {
        kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(wb, gb, momentum, n, lr, mu, weight_decay);
    };
    if (momentum != nullptr)
        wide ? go(sgd_bf16_kernel<true, true>) : go(sgd_bf16_kernel<true, false>);
    else
        wide ? go(sgd_bf16_kernel<false, true>) : go(sgd_bf16_kernel<false, false>);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_mse_bf16(const void* y, const void* target, void* dy, float* loss_out, uint64_t n,
                            float scale, cudaStream_t stream) {
    if (n == 0)
        return cudaSuccess;
    uint64_t blocks = (n + 256 * 8 - 1) / (256 * 8);
    if (blocks > 148 * 8)
        blocks = 148 * 8;
    const uintptr_t bits = reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(target) |
                           reinterpret_cast<uintptr_t>(dy);
    mse_bf16_kernel<<<static_cast<int>(blocks), 256, 0, stream>>>(
            static_cast<const __nv_bfloat16*>(y), static_cast<const __nv_bfloat16*>(target),
            static_cast<__nv_bfloat16*>(dy), loss_out, n, scale, (bits & 15) == 0 ? 1 : 0);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_add_rmsnorm_bf16(const void* x, const void* y, void* x_out, void* n_out, float* inv_rms,
                                    int rows, int cols, float eps, cudaStream_t stream) {
    if (rows <= 0)
        return cudaSuccess;
    if (cols <= 0 || cols % 8 || cols > kNormThreads * kNormMaxVec * 8)
        return cudaErrorInvalidValue;
    auto go = [&](auto kernel) {
        kernel<<<rows, kNormThreads, 0, stream>>>(static_cast<const uint4*>(x), static_cast<const uint4*>(y),
                                                  static_cast<uint4*>(x_out), static_cast<uint4*>(n_out), inv_rms,
                                                  cols, eps);
    };
    switch (norm_nv(cols)) {
        case 1: go(add_rmsnorm_kernel<1>); break;
        case 2: go(add_rmsnorm_kernel<2>); break;
        case 4: go(add_rmsnorm_kernel<4>); break;
        default: go(add_rmsnorm_kernel<8>); break;
    }
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_rmsnorm_bwd_bf16(const void* dn, const void* n, const float* inv_rms, const void* dres,
                                    void* dx, int rows, int cols, cudaStream_t stream) {
    if (rows <= 0)
        return cudaSuccess;
    if (cols <= 0 || cols % 8 || cols > kNormThreads * kNormMaxVec * 8)
        return cudaErrorInvalidValue;
    auto go = [&](auto kernel) {
        kernel<<<rows, kNormThreads, 0, stream>>>(static_cast<const uint4*>(dn), static_cast<const uint4*>(n),
                                                  inv_rms, static_cast<const uint4*>(dres),
                                                  static_cast<uint4*>(dx), cols);
    };
    switch (norm_nv(cols)) {
        case 1: go(rmsnorm_bwd_kernel<1>); break;
        case 2: go(rmsnorm_bwd_kernel<2>); break;
        case 4: go(rmsnorm_bwd_kernel<4>); break;
        default: go(rmsnorm_bwd_kernel<8>); break;
    }
    count_launch();
    return cudaGetLastError();
}

}  // namespace ew
}  // namespace mgk
