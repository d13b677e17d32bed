"""Products whose rows are grouped by expert, on the persistent kernel's tiles, against float64: tiles of one
128-row block, and tiles of several blocks of one group out of the row-tile list."""
import pytest
import torch
from gemm_check import BLOCKS, check, check_dswiglu, mk, product

pytestmark = pytest.mark.gpu


def blocks_of(blocks, **kw):
    return dict(m_block_group=torch.tensor(blocks, device="cuda", dtype=torch.int32), **kw)


def rows_of(blocks):
    """(group, rows) of each run of blocks of one group."""
    first = 0
    for i in range(1, len(blocks) + 1):
        if i == len(blocks) or blocks[i] != blocks[first]:
            yield blocks[first], slice(128 * first, 128 * i)
            first = i


def spoil_padding(x, blocks):
    """NaN and infinity in the rows of padding blocks: a tile may load them, no result may show them."""
    for g, r in rows_of(blocks):
        if g < 0:
            x[r] = float("nan")
            x[r.start] = float("inf")
    return x


def untouched(*results):
    return all(bool((t == 7.0).all()) for t in results)


@pytest.mark.parametrize("variant", [1, 2, 3])
@pytest.mark.parametrize("blocks", BLOCKS)
def test_grouped_rows_on_tiles_of_several_blocks(variant, blocks):
    from megray_b200.ops import EPI_SWIGLU, gemm

    torch.manual_seed(4)
    E, N, K, M = 3, 264, 192, 128 * len(blocks)
    groups = blocks_of(blocks, groups=E, variant=variant)
    x, w, wgu = spoil_padding(mk(M, K), blocks), mk(E * N, K), mk(E * 2 * N, K)
    out = torch.full((M, N), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm(x, w, out, n=N, group_rows_b=N, **groups)
    gu = torch.full((M, 2 * N), 7.0, device="cuda", dtype=torch.bfloat16)
    h = torch.full((M, N), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm(x, wgu, gu, out2=h, n=N, epilogue=EPI_SWIGLU, group_rows_b=2 * N, **groups)
    for e, r in rows_of(blocks):
        if e < 0:  # padding blocks are left untouched
            assert untouched(out[r], gu[r], h[r])
        else:
            check(out[r], *product(x[r], w[e * N:(e + 1) * N], False, False), K)
            check(gu[r], *product(x[r], wgu[e * 2 * N:(e + 1) * 2 * N], False, False), K)


@pytest.mark.parametrize("variant", [1, 2, 3])
@pytest.mark.parametrize("blocks", BLOCKS)
def test_grouped_rows_against_transposed_weights(variant, blocks):
    """The two products of the MoE backward: weights stored [K, N] per group, with and without the SwiGLU
    derivative."""
    from megray_b200.ops import EPI_DSWIGLU, gemm

    torch.manual_seed(6)
    E, N, K, M = 3, 264, 192, 128 * len(blocks)
    groups = blocks_of(blocks, groups=E, variant=variant, group_rows_b=K)
    dy, w, gu = spoil_padding(mk(M, K), blocks), mk(E * K, N, 0.1), spoil_padding(mk(M, 2 * N), blocks)
    out = torch.full((M, N), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm(dy, w, out, b_mn=True, n=N, **groups)
    dgu = torch.full((M, 2 * N), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm(dy, w, dgu, b_mn=True, epilogue=EPI_DSWIGLU, aux=gu, n=N, **groups)
    for e, r in rows_of(blocks):
        if e < 0:
            assert untouched(out[r], dgu[r])
        else:
            dh, mass = product(dy[r], w[e * K:(e + 1) * K], False, True)
            check(out[r], dh, mass, K)
            check_dswiglu(dgu[r], gu[r], dh, mass, K)


@pytest.mark.parametrize("blocks", [
    [0] * 120 + [1] + [2] + [3] * 2 + [-1] * 4,        # one group holds nearly all rows
    [i // 3 for i in range(192)] + [-1] * 8,           # many groups of three blocks
    [0] * 300 + [1] + [2] * 402 + [-1],                # as many blocks as the row-tile list has entries for
    [0] * 300 + [1] + [2] * 402 + [-1] * 2,            # one more: tiles of one block
])
def test_automatic_choice_for_grouped_rows(blocks):
    from megray_b200.ops import gemm

    torch.manual_seed(7)
    E, N, K, M = max(blocks) + 1, 512, 72, 128 * len(blocks)
    x, w = spoil_padding(mk(M, K), blocks), mk(E * N, K)
    out = torch.full((M, N), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm(x, w, out, n=N, group_rows_b=N, **blocks_of(blocks, groups=E))
    for e, r in rows_of(blocks):
        if e < 0:
            assert untouched(out[r])
        else:
            check(out[r], *product(x[r], w[e * N:(e + 1) * N], False, False), K)


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
