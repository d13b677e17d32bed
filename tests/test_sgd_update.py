"""The SGD kernel at the edges of its 16-element groups and blocks, on buffers that allow 256-bit accesses
and on ones that start 16 bytes later, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 16, 17, 4096, 4097, 8192 + 31, 300_007])
@pytest.mark.parametrize("shift", [0, 8])
@pytest.mark.parametrize("momentum", [0.0, 0.9])
def test_update(n, shift, momentum):
    from megray_b200.ops import sgd_step

    torch.manual_seed(n)
    w, g = (torch.randn(n + 16, device="cuda").to(torch.bfloat16)[shift:shift + n] for _ in range(2))
    m = torch.randn(n + 16, device="cuda")[shift // 2:shift // 2 + n] if momentum else None
    lr, wd = 0.1, 0.01
    w0, step = w.double(), g.double() + wd * w.double()
    if m is not None:
        step = momentum * m.double() + step
    sgd_step(w, g, lr, m, momentum, wd)
    want = w0 - lr * step
    size = w0.abs() + g.double().abs() + step.abs()  # float32 terms: a few 2^-23 of these; then bf16
    assert bool(((w.double() - want).abs() <= want.abs() * 2.0 ** -8 + size * 2.0 ** -21).all())
    if m is not None:
        assert bool(((m.double() - step).abs() <= (size + step.abs()) * 2.0 ** -21).all())
