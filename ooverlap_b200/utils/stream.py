"""The current CUDA stream as a plain integer."""
from __future__ import annotations

import torch


def current_stream_ptr() -> int:
    """``cudaStream_t`` of the current stream of the current device.  ``torch.cuda.current_stream().cuda_stream`` builds a
    Python stream object on the way, which costs more than the rest of a launch's bookkeeping."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())
