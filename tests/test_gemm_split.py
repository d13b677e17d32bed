"""The small-tile / cluster split-K kernel against float64 at the sizes where it can go wrong: edges of
tiles, remainders of K, more CTAs than k-steps, every operand layout and epilogue."""
import pytest
import torch
from gemm_check import BLOCKS, check, check_dswiglu, mk, product

pytestmark = pytest.mark.gpu


PLANS = [64 + 1, 64 + 2, 64 + 8, 128 + 1, 128 + 4, 128 + 8, 256 + 1, 256 + 2, 256 + 8]


@pytest.mark.parametrize("variant", PLANS)
@pytest.mark.parametrize("M,N,K", [(8, 8, 8), (128, 64, 64), (136, 72, 136), (304, 264, 520), (256, 512, 2048)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
def test_products(variant, M, N, K, a_mn, b_mn):
    from megray_b200.ops import EPI_ACCUM, EPI_STORE_F32, gemm

    torch.manual_seed(M + N + K)
    a, b = mk(K, M) if a_mn else mk(M, K), mk(K, N) if b_mn else mk(N, K)
    want, mass = product(a, b, a_mn, b_mn)
    kw = dict(a_mn=a_mn, b_mn=b_mn, variant=variant)
    got = gemm(a, b, **kw)
    check(got, want, mass, K)
    assert torch.equal(got, gemm(a, b, **kw))  # a fixed order of summation
    check(gemm(a, b, epilogue=EPI_STORE_F32, **kw), want, mass, K, rounded=False)
    d = mk(M, N)
    want = want + d.double()
    check(gemm(a, b, d, epilogue=EPI_ACCUM, **kw), want, mass + want.abs(), K + 1)


@pytest.mark.parametrize("variant", [64 + 1, 64 + 4, 128 + 1, 128 + 8, 256 + 1, 256 + 8])
@pytest.mark.parametrize("M,F,K", [(1, 32, 64), (130, 72, 200), (256, 384, 1024)])
def test_swiglu_and_its_derivative(variant, M, F, K):
    from megray_b200.ops import EPI_DSWIGLU, EPI_SWIGLU, gemm

    torch.manual_seed(3)
    x, w = mk(M, K), mk(2 * F, K, 0.1)
    gu, h = gemm(x, w, epilogue=EPI_SWIGLU, n=F, variant=variant)
    want, mass = product(x, w, False, False)
    check(gu, want, mass, K)
    g, u = want[:, :F], want[:, F:]
    s = torch.sigmoid(g)
    # |d silu| <= 1.1 |dg|; a few 2^-20 for the fast exponential and division
    check(h, g * s * u, 1.1 * (mass[:, :F] * u.abs() + mass[:, F:] * (g * s).abs()) + (g * s * u).abs(), K + 16)
    dy, wd = mk(M, K), mk(K, F, 0.1)
    dgu = gemm(dy, wd, b_mn=True, epilogue=EPI_DSWIGLU, aux=gu, n=F, variant=variant)
    dh, mass = product(dy, wd, False, True)
    check_dswiglu(dgu, gu, dh, mass, K)


def test_a_shape_the_kernel_does_not_take_is_refused():
    from megray_b200.ops import gemm

    a, b = mk(64, 64), mk(64, 64)
    for variant in (64 + 3, 64 + 16, 192 + 1):
        with pytest.raises(RuntimeError):
            gemm(a, b, variant=variant)


@pytest.mark.parametrize("variant", [64 + 2, 256 + 1])
@pytest.mark.parametrize("blocks", BLOCKS)
def test_grouped_rows(variant, blocks):
    from megray_b200.ops import EPI_SWIGLU, gemm

    torch.manual_seed(4)
    E, N, K, M = 3, 264, 192, 128 * len(blocks)
    groups = dict(m_block_group=torch.tensor(blocks, device="cuda", dtype=torch.int32), groups=E, variant=variant)
    x, w, wgu = mk(M, K), mk(E * N, K), mk(E * 2 * N, K)
    out = torch.full((M, N), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm(x, w, out, n=N, group_rows_b=N, **groups)
    gu = torch.full((M, 2 * N), 7.0, device="cuda", dtype=torch.bfloat16)
    h = torch.full((M, N), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm(x, wgu, gu, out2=h, n=N, epilogue=EPI_SWIGLU, group_rows_b=2 * N, **groups)
    for i, e in enumerate(blocks):
        r = slice(128 * i, 128 * (i + 1))
        if e < 0:  # padding blocks are left untouched
            assert all(float((t[r].float() - 7.0).abs().max()) == 0.0 for t in (out, gu, h))
        else:
            check(out[r], *product(x[r], w[e * N:(e + 1) * N], False, False), K)
            check(gu[r], *product(x[r], wgu[e * 2 * N:(e + 1) * 2 * N], False, False), K)


@pytest.mark.parametrize("variant", [64 + 4, 128 + 1, 256 + 2])
@pytest.mark.parametrize("blocks", BLOCKS)
def test_grouped_rows_against_transposed_weights(variant, blocks):
    from megray_b200.ops import EPI_DSWIGLU, gemm

    torch.manual_seed(6)
    E, N, K, M = 3, 264, 192, 128 * len(blocks)
    groups = dict(m_block_group=torch.tensor(blocks, device="cuda", dtype=torch.int32), groups=E, variant=variant,
                  group_rows_b=K)
    dy, w, gu = mk(M, K), mk(E * K, N, 0.1), mk(M, 2 * N)
    out = torch.full((M, N), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm(dy, w, out, b_mn=True, n=N, **groups)
    dgu = torch.full((M, 2 * N), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm(dy, w, dgu, b_mn=True, epilogue=EPI_DSWIGLU, aux=gu, n=N, **groups)
    for i, e in enumerate(blocks):
        r = slice(128 * i, 128 * (i + 1))
        if e < 0:
            assert all(bool((t[r] == 7.0).all()) for t in (out, dgu))
        else:
            dh, mass = product(dy[r], w[e * K:(e + 1) * K], False, True)
            check(out[r], dh, mass, K)
            check_dswiglu(dgu[r], gu[r], dh, mass, K)


@pytest.mark.parametrize("variant", [64 + 4, 128 + 2])
def test_grouped_k_ranges(variant):
    from megray_b200.ops import gemm

    torch.manual_seed(5)
    E, M, N, T = 4, 512, 200, 896
    kb, ke = [0, 128, 128, 640], [128, 128, 640, 896]  # group 1 is empty: zeros
    dy, x = mk(T, M), mk(T, N)
    out = gemm(dy, x, a_mn=True, b_mn=True, groups=E, variant=variant,
               k_begin=torch.tensor(kb, device="cuda", dtype=torch.int32),
               k_end=torch.tensor(ke, device="cuda", dtype=torch.int32))
    for e in range(E):
        check(out[e * M:(e + 1) * M], *product(dy[kb[e]:ke[e]], x[kb[e]:ke[e]], True, True), T)
