"""Row tiles of grouped problems, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def mk(r, c, scale=0.5):
    return (torch.randn(r, c, device="cuda") * scale).to(torch.bfloat16)


def product(a, b, a_mn, b_mn):
    """(A B^T, |A| |B|^T) in float64."""
    a, b = a.double(), b.double()
    a, b = (a.t() if a_mn else a), (b if b_mn else b.t())
    return a @ b, a.abs() @ b.abs()


def check(got, want, mass, k, rounded=True):
    """float32 sums of k products in any order are within k * 2^-24 of the sum of their magnitudes
    (twice that here); a bf16 result is rounded once more, by at most 2^-8 of its value."""
    from megray_b200.ops import gemm_error_flag

    torch.cuda.synchronize()
    assert int(gemm_error_flag().item()) == 0
    bound = mass * (k * 2.0 ** -23) + (want.abs() * 2.0 ** -8 if rounded else 0) + 1e-30
    assert bool(((got.double() - want).abs() <= bound).all())


BLOCKS = [
    [0, 0, 0, 1, -1, 2, 2, 2, 2, 2, -1, -1],
    [1] * 31 + [0] * 3 + [2] * 34 + [-1] * 3,  # runs across the 32-block batches of the list's builder
    [-1, -1, 2],
    [-1, -1],
]


@pytest.mark.parametrize("variant", [2, 3])
@pytest.mark.parametrize("blocks", BLOCKS)
def test_grouped_rows_on_tiles_of_several_blocks(variant, blocks):
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


@pytest.mark.parametrize("variant", [0, 2, 3])
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
