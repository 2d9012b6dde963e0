"""torch plumbing shared by the op mirrors: argument checks, dtype codes, stream and workspace."""
from __future__ import annotations

import torch

from . import _lib

_DT = {torch.float16: _lib.F16, torch.bfloat16: _lib.BF16, torch.float32: _lib.F32}


def dtype_code(t: torch.dtype) -> int:
    if t not in _DT:
        raise RuntimeError(f"unsupported dtype {t}")
    return _DT[t]


def require_cuda(*tensors: torch.Tensor) -> torch.device:
    dev = None
    for t in tensors:
        if t is None:
            continue
        if not t.is_cuda:
            raise RuntimeError("b200 nvfp4 ops take CUDA tensors only (there is no CPU path)")
        if dev is None:
            dev = t.device
        elif t.device != dev:
            raise RuntimeError("all tensors must be on the same device")
    return dev


def require(cond: bool, msg: str) -> None:
    if not cond:
        raise RuntimeError(msg)


def stream_ptr(device: torch.device) -> int:
    return torch.cuda.current_stream(device).cuda_stream


WS_SHARED, WS_LINEAR, WS_ROUTER, WS_GEMM = 0, 1, 2, 3       # slots of a stream's scratch (csrc/torch_host.cpp)


def workspace(device: torch.device, nbytes: int, slot: int = WS_SHARED) -> torch.Tensor:
    """Grow-only scratch buffer per (device, current stream, slot), shared with the native host path.  Calls issued on one
    stream serialise on the GPU, so sharing it between consecutive ops is safe; its address is stable once large enough,
    which CUDA-graph capture relies on."""
    return _lib.host().workspace(torch.cuda.current_device() if device.index is None else device.index, nbytes, slot)


def status_word(device, slot: int) -> int:
    """The first int of a slot's scratch, where the ops that use it leave their status word.  Synchronises the device."""
    dev = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    torch.cuda.synchronize(dev)
    return int(workspace(dev, 256, slot)[:4].view(torch.int32).item())


def ptr(t) -> int:
    return 0 if t is None else t.data_ptr()
