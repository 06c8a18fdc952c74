"""Host side of the byte histogram: the plugin entry of the reference's second task.

``custom_kernel((data, output))`` has the signature the task defines
(pmpp_v2/histogram_py/task.py:4-5; submission entry pmpp_v2/histogram_py/submission_v1.py:110-113):
``data`` uint8 ``[size]`` on the GPU, ``output`` int64 ``[256]`` preallocated by the caller; the counts
are written into ``output`` and it is returned.  All work is in liba2a.so (``a2a_histogram256``);
there is no CPU or PyTorch fallback.
"""
from __future__ import annotations

from typing import Tuple

import torch

from . import _lib

NUM_BINS = 256


def histogram256(data: torch.Tensor, output: torch.Tensor) -> torch.Tensor:
    """Counts of the byte values of ``data`` into ``output`` on the current stream; returns ``output``."""
    out = _lib.host().histogram(data, output)
    if out is not None:
        return out if type(out) is not int else _lib.check(out)
    # something is wrong, or unusual: look again, one thing at a time
    if data.dtype is not torch.uint8 or not data.is_cuda or not data.is_contiguous() or data.dim() != 1:
        raise _lib.A2AError(_lib.A2A_ERR_CONFIG, "data must be a contiguous 1-D uint8 CUDA tensor, got "
                            f"{data.dtype} {tuple(data.shape)} on {data.device}")
    device = data.get_device()
    if (output.dtype is not torch.int64 or output.numel() != NUM_BINS or not output.is_contiguous()
            or not output.is_cuda or output.get_device() != device):
        raise _lib.A2AError(_lib.A2A_ERR_CONFIG, f"output must be a contiguous int64 [{NUM_BINS}] tensor on {data.device}")
    if device != torch.cuda.current_device():
        with torch.cuda.device(device):
            return histogram256(data, output)
    rc = _lib.load().a2a_histogram256(data.data_ptr(), data.numel(), output.data_ptr(), _lib.current_stream())
    if rc != 0:
        _lib.check(rc)
    return output


def custom_kernel(data: Tuple[torch.Tensor, torch.Tensor]) -> torch.Tensor:
    values, output = data
    return histogram256(values, output)
