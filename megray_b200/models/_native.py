"""Operands of the native one-call passes (src/capi/step_c.cpp)."""
from __future__ import annotations

import torch


def plain(t, shape, dtype=torch.bfloat16) -> int:
    """Device address of a contiguous, 16-byte aligned CUDA tensor of this shape and type; 0 for
    anything else (which the op-by-op path takes or refuses)."""
    if (not isinstance(t, torch.Tensor) or t.dtype is not dtype or t.shape != shape or not t.is_contiguous() or
            not t.is_cuda):
        return 0
    p = t.data_ptr()
    return 0 if p & 15 else p
