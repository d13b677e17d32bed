// One pass of the single-GPU models as one native call each: the same launches, in the same order
// and with the same arguments as the op-by-op Python methods (megray_b200/models), without the
// 8-12 us of interpreter and ctypes time in front of every launch.  At small sizes that time, not
// the GPU, was the length of a step.  Nothing is kept between calls: every pointer comes with the
// call.
#include "kernels/collectives.cuh"
#include "kernels/elementwise.cuh"
#include "kernels/gemm_tcgen05.cuh"
#include "kernels/moe.cuh"
#include "megray/c_api.h"

namespace {

using mgk::gemm::GemmArgs;

// The first error ends the sequence.
struct Seq {
    cudaStream_t stream;
    int* error_flag;
    cudaError_t err = cudaSuccess;

    void operator()(cudaError_t e) {
        if (err == cudaSuccess)
            err = e;
    }
    bool ok() const { return err == cudaSuccess; }
    int rc() const { return err == cudaSuccess ? 0 : -static_cast<int>(err); }

    // contiguous operands: a is [M, K] (or [K, M]), b [N, K] (or [K, N])
    GemmArgs args(const void* a, bool a_mn, const void* b, bool b_mn, void* d, int M, int N, int K, int epilogue) const {
        GemmArgs g{};
        g.A = a;
        g.B = b;
        g.D = d;
        g.M = M;
        g.N = N;
        g.K = K;
        g.lda = a_mn ? M : K;
        g.ldb = b_mn ? N : K;
        const bool pair = epilogue == mgk::gemm::EPI_SWIGLU || epilogue == mgk::gemm::EPI_DSWIGLU;
        g.ldd = pair ? 2 * N : N;
        g.aux_off = pair ? N : 0;
        g.a_mn = a_mn;
        g.b_mn = b_mn;
        g.epilogue = epilogue;
        g.error_flag = error_flag;
        return g;
    }
    void gemm(const GemmArgs& g) {
        if (ok())
            (*this)(mgk::gemm::launch_gemm_bf16(g, stream));
    }
};

// out[M, N] = a^T b over K rows, cut into `splits` K ranges when the tiles of the output fill the
// chip badly (float32 partials in `ws`, summed in float32)
void wgrad(Seq& s, const void* a, const void* b, void* out, int M, int N, int K, const megray_k_split& split, void* ws) {
    using namespace mgk::gemm;
    if (split.splits <= 1) {
        s.gemm(s.args(a, true, b, true, out, M, N, K, EPI_STORE));
        return;
    }
    GemmArgs g = s.args(a, true, b, true, ws, M, N, K, EPI_STORE_F32);
    g.variant = M % 512 == 0 ? 3 : 2;
    g.grouped.k_begin = split.k_begin;
    g.grouped.k_end = split.k_end;
    g.grouped.groups = split.splits;
    s.gemm(g);
    const void* part[8];
    for (int i = 0; i < split.splits && i < 8; ++i)
        part[i] = static_cast<const float*>(ws) + static_cast<size_t>(i) * M * N;
    if (s.ok())
        s(mgk::coll::launch_reduce_n(part, split.splits, out, static_cast<uint64_t>(M) * N, MegRay::MEGRAY_FLOAT32,
                                     MegRay::MEGRAY_BFLOAT16, MegRay::MEGRAY_SUM, 1.0f, s.stream));
}

}  // namespace

extern "C" {

int megray_mlp_forward(const megray_mlp_args* a, const void* x, void* stream) {
    using namespace mgk;
    using namespace mgk::gemm;
    if (a == nullptr || x == nullptr || a->layers < 1)
        return 6;
    Seq s{static_cast<cudaStream_t>(stream), a->error_flag};
    const int T = a->tokens, d = a->d_model, f = a->ffn;
    s(ew::launch_add_rmsnorm_bf16(x, nullptr, nullptr, a->layer[0].xg, a->layer[0].inv_rms, T, d, 1e-6f, s.stream));
    for (int l = 0; l < a->layers && s.ok(); ++l) {
        const megray_mlp_layer& w = a->layer[l];
        GemmArgs up = s.args(w.xg, false, w.w_gu, false, w.gu, T, f, d, EPI_SWIGLU);
        up.D2 = w.h;
        up.ldd2 = f;
        s.gemm(up);
        s.gemm(s.args(w.h, false, w.w_down, false, a->y, T, d, f, EPI_STORE));
        const bool last = l + 1 == a->layers;
        if (s.ok())
            s(ew::launch_add_rmsnorm_bf16(x, a->y, a->xs[l & 1], last ? nullptr : a->layer[l + 1].xg,
                                          last ? nullptr : a->layer[l + 1].inv_rms, T, d, 1e-6f, s.stream));
        x = a->xs[l & 1];
    }
    return s.rc();
}

int megray_mlp_backward(const megray_mlp_args* a, const void* dy, void* stream) {
    using namespace mgk;
    using namespace mgk::gemm;
    if (a == nullptr || dy == nullptr || a->layers < 1)
        return 6;
    Seq s{static_cast<cudaStream_t>(stream), a->error_flag};
    const int T = a->tokens, d = a->d_model, f = a->ffn;
    for (int l = a->layers - 1; l >= 0 && s.ok(); --l) {
        const megray_mlp_layer& w = a->layer[l];
        GemmArgs g = s.args(dy, false, w.w_down, true, a->dgu, T, f, d, EPI_DSWIGLU);
        g.aux = w.gu;
        g.ldaux = 2 * f;
        s.gemm(g);
        wgrad(s, dy, w.h, w.g_down, d, f, T, a->split_down, a->wgrad_ws);
        s.gemm(s.args(a->dgu, false, w.w_gu, true, a->dn, T, d, 2 * f, EPI_STORE));
        wgrad(s, a->dgu, w.xg, w.g_gu, 2 * f, d, T, a->split_gu, a->wgrad_ws);
        if (s.ok())
            s(ew::launch_rmsnorm_bwd_bf16(a->dn, w.xg, w.inv_rms, dy, a->dres[l & 1], T, d, s.stream));
        dy = a->dres[l & 1];
    }
    return s.rc();
}

int megray_moe_forward(const megray_moe_args* a, const void* x, const float* logits, void* stream) {
    using namespace mgk;
    using namespace mgk::gemm;
    if (a == nullptr || x == nullptr || logits == nullptr)
        return 6;
    Seq s{static_cast<cudaStream_t>(stream), a->error_flag};
    const int T = a->tokens, E = a->experts, H = a->hidden, F = a->ffn, cap = a->capacity;
    moe::PeerBufs xp{}, yp{};
    xp.p[0] = a->x_perm;
    yp.p[0] = a->y_perm;
    s(cudaMemsetAsync(a->counts, 0, sizeof(int) * E, s.stream));
    if (s.ok())
        s(moe::launch_route(logits, T, E, a->idx, a->w, a->counts, s.stream));
    if (s.ok())
        s(moe::launch_plan(a->counts, 1, 0, E, cap,
                           moe::PlanOut{a->send_base, a->seg_begin, a->seg_end, a->seg_rows, a->block_group, a->total},
                           s.stream));
    if (s.ok())
        s(moe::launch_zero_pads(a->x_perm, H, a->seg_begin, a->seg_rows, a->seg_end, E, s.stream));
    if (s.ok())
        s(cudaMemsetAsync(a->cursor, 0, sizeof(int) * E, s.stream));
    if (s.ok())
        s(moe::launch_dispatch(x, T, H, a->idx, nullptr, a->send_base, a->cursor, nullptr, a->pos, xp, E, E, cap, s.stream));
    GemmArgs up = s.args(a->x_perm, false, a->w_gu, false, a->gu, cap, F, H, EPI_SWIGLU);
    up.D2 = a->h;
    up.ldd2 = F;
    up.grouped = GroupedArgs{a->block_group, 2 * F, nullptr, nullptr, E};
    s.gemm(up);
    GemmArgs down = s.args(a->h, false, a->w_down, false, a->y_perm, cap, H, F, EPI_STORE);
    down.grouped = GroupedArgs{a->block_group, H, nullptr, nullptr, E};
    s.gemm(down);
    if (s.ok())
        s(moe::launch_combine(a->out, T, H, a->idx, a->w, a->pos, yp, E, cap, s.stream));
    return s.rc();
}

int megray_moe_backward(const megray_moe_args* a, const void* dout, void* stream) {
    using namespace mgk;
    using namespace mgk::gemm;
    if (a == nullptr || dout == nullptr)
        return 6;
    Seq s{static_cast<cudaStream_t>(stream), a->error_flag};
    const int T = a->tokens, E = a->experts, H = a->hidden, F = a->ffn, cap = a->capacity;
    moe::PeerBufs yp{}, dyp{}, dxp{};
    yp.p[0] = a->y_perm;
    dyp.p[0] = a->dy_perm;
    dxp.p[0] = a->dx_perm;
    s(moe::launch_combine_dw(dout, T, H, a->idx, a->pos, yp, E, cap, a->dw, s.stream));
    if (s.ok())
        s(moe::launch_zero_pads(a->dy_perm, H, a->seg_begin, a->seg_rows, a->seg_end, E, s.stream));
    if (s.ok())
        s(moe::launch_dispatch(dout, T, H, a->idx, a->w, a->send_base, a->cursor, a->pos, a->pos, dyp, E, E, cap, s.stream));
    GemmArgs g = s.args(a->dy_perm, false, a->w_down, true, a->dgu, cap, F, H, EPI_DSWIGLU);
    g.aux = a->gu;
    g.ldaux = 2 * F;
    g.grouped = GroupedArgs{a->block_group, H, nullptr, nullptr, E};
    s.gemm(g);
    GemmArgs wd = s.args(a->dy_perm, true, a->h, true, a->g_down, H, F, cap, EPI_STORE);
    wd.grouped = GroupedArgs{nullptr, 0, a->seg_begin, a->seg_end, E};
    s.gemm(wd);
    GemmArgs dx = s.args(a->dgu, false, a->w_gu, true, a->dx_perm, cap, H, 2 * F, EPI_STORE);
    dx.grouped = GroupedArgs{a->block_group, 2 * F, nullptr, nullptr, E};
    s.gemm(dx);
    GemmArgs wg = s.args(a->dgu, true, a->x_perm, true, a->g_gu, 2 * F, H, cap, EPI_STORE);
    wg.grouped = GroupedArgs{nullptr, 0, a->seg_begin, a->seg_end, E};
    s.gemm(wg);
    if (s.ok())
        s(moe::launch_combine(a->dx, T, H, a->idx, nullptr, a->pos, dxp, E, cap, s.stream));
    if (s.ok())
        s(moe::launch_route_bwd(a->idx, a->w, a->dw, T, E, a->dlogits, s.stream));
    return s.rc();
}

}  // extern "C"
