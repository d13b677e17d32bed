"""The SGD update refuses buffers that its vector accesses cannot read, before anything is launched."""
import ctypes as C

import pytest
import torch

INVALID_VALUE = -1


def call(n, w=0, g=0, m=None):
    """The return code for three host buffers at these byte offsets from a 64-byte boundary."""
    from megray_b200 import _lib

    buf = C.create_string_buffer(4096)
    base = (C.addressof(buf) + 63) // 64 * 64
    return _lib.load().megray_sgd_bf16(base + w, base + 1024 + g, None if m is None else base + 2048 + m, n, 0.1, 0.9,
                                       0.0, None)


@pytest.mark.skipif(torch.cuda.is_available(), reason="host buffers: only where nothing can be launched")
def test_misaligned_buffers_are_an_argument_error():
    for n in (16, 17, 64):
        for m in (4, 8, 12, 20):  # groups of 16 elements read the momentum 16 bytes at a time
            assert call(n, m=m) == INVALID_VALUE
    assert call(64, m=2) == INVALID_VALUE and call(1, m=2) == INVALID_VALUE
    assert call(64, w=8) == INVALID_VALUE and call(64, g=4) == INVALID_VALUE
    # everything else gets as far as the launch, which fails here for want of a device
    for n in (1, 15):
        assert call(n, m=4) not in (0, INVALID_VALUE)  # single elements only
    for m in (0, 16, None):
        assert call(64, m=m) not in (0, INVALID_VALUE)
    assert call(64, w=16, m=32) not in (0, INVALID_VALUE)


@pytest.mark.gpu
def test_a_momentum_view_off_the_boundary():
    from megray_b200.ops import sgd_step

    w, g = (torch.randn(64, device="cuda").to(torch.bfloat16) for _ in range(2))
    m = torch.zeros(68, device="cuda")
    before = w.clone()
    with pytest.raises(RuntimeError):
        sgd_step(w, g, 0.1, m[1:65], 0.9)
    assert torch.equal(w, before)
    sgd_step(w[:15], g[:15], 0.1, m[1:16], 0.9)
    assert torch.equal(m[1:16], g[:15].float()) and torch.equal(w[15:], before[15:])
