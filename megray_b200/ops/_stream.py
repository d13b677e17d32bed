"""The current CUDA stream as the handle the native library takes."""
import torch


def raw_stream() -> int:
    """``torch.cuda.current_stream().cuda_stream`` without building a Stream object."""
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device())
