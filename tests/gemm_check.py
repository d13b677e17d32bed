"""Products of the GEMM tests in float64 and the bounds their results have to keep."""
import torch

# groups of the 128-row blocks of grouped problems; -1 = padding block
BLOCKS = [
    [0, 0, 0, 1, -1, 2, 2, 2, 2, 2, -1, -1],
    [1] * 31 + [0] * 3 + [2] * 34 + [-1] * 3,  # runs across the 32-block batches in which a row-tile list is built
    [-1, -1, 2],
    [-1, -1],
]


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


def check_dswiglu(dgu, gu, dh, mass, k):
    """The gradient of silu(g) * u for dh (with the magnitudes ``mass`` of its k products) and the saved
    rounded g and u, which both sides read; the factors are formed in float32 (16 * 2^-23)."""
    f = dh.shape[1]
    g, u = gu[:, :f].double(), gu[:, f:].double()
    s = torch.sigmoid(g)
    want = torch.cat([dh * u * (s + g * s * (1 - s)), dh * g * s], 1)
    scale = torch.cat([u.abs() * (s + g.abs() * s * (1 - s)), (g * s).abs()], 1)
    check(dgu, want, scale * torch.cat([mass, mass], 1), k + 16)
