"""Mirrors of the dense NVFP4 ops the reference enables in vLLM (`torch.ops._C.*` wrappers in
vllm/_custom_ops.py), backed by libb200nvfp4.so."""
from __future__ import annotations

import torch

from . import _lib
from ._torch_util import WS_GEMM, WS_LINEAR, status_word


def scaled_fp4_quant(input: torch.Tensor, input_global_scale: torch.Tensor, is_sf_swizzled_layout: bool = True):
    """bf16/f16 [M,K] -> (packed E2M1 codes u8 [M,K/2], E4M3 block scales).

    Mirrors scaled_fp4_quant (vllm/_custom_ops.py:1600-1671).  Scales come back as float8_e4m3fn:
    [round_up(M,128), round_up(K/16,4)] in the 128x4 swizzled tile layout (default) or [M, K/16]
    linear when is_sf_swizzled_layout is False.  input_global_scale is a one-element f32 CUDA tensor."""
    return _lib.host().scaled_fp4_quant(input, input_global_scale, is_sf_swizzled_layout)


def cutlass_scaled_fp4_mm(a: torch.Tensor, b: torch.Tensor, block_scale_a: torch.Tensor, block_scale_b: torch.Tensor,
                          alpha: torch.Tensor, out_dtype: torch.dtype, *, out: torch.Tensor | None = None,
                          tile_n: int = 0) -> torch.Tensor:
    """out[M,N] = alpha * (a . block_scale_a)(b . block_scale_b)^T on the tcgen05 tensor cores.

    Mirrors cutlass_scaled_fp4_mm (vllm/_custom_ops.py:741-753): a [M,K/2] and b [N,K/2] packed E2M1
    bytes, block scales in the swizzled 128x4 layout as produced by scaled_fp4_quant, alpha a
    one-element f32 CUDA tensor, out_dtype bf16 or f16.  Pass `out` to write in place like the raw
    torch.ops._C op does."""
    return _lib.host().cutlass_scaled_fp4_mm(a, b, block_scale_a, block_scale_b, alpha, out_dtype, out, tile_n)


def nvfp4_linear(x: torch.Tensor, x_global_scale: torch.Tensor, w_codes: torch.Tensor, w_block_scale: torch.Tensor,
                 alpha: torch.Tensor, *, out: torch.Tensor | None = None, tile_n: int = 0) -> torch.Tensor:
    """y[M,N] = alpha * NVFP4(x) @ W^T: scaled_fp4_quant followed by cutlass_scaled_fp4_mm in ONE library call
    (b200fp4_linear_nvfp4), which is what a quantized linear layer does on every forward (the pair of ops in vLLM's
    NVFP4 linear apply, nvfp4_utils.py; emulated by the reference at fix_nvfp4_emulation_backend.py:60-102).  Same codes
    and products as calling the two ops (for few tokens the f32 sums over K may be grouped otherwise); the launches are a few
    microseconds apart instead of a Python call apart, and for few tokens it is one kernel that quantizes its own operand.
    x [M,K] bf16/f16 (rows may be strided), w_codes [N,K/2] u8, w_block_scale swizzled, alpha / x_global_scale one f32."""
    return _lib.host().nvfp4_linear(x, x_global_scale, w_codes, w_block_scale, alpha, out, tile_n)


def last_gemm_status(device=None) -> int:
    """Status word of the most recent GEMM op on the current stream of `device` (0 = ok) or, where that is 0, of the most recent
    nvfp4_linear.  Synchronises."""
    return status_word(device, WS_GEMM) or status_word(device, WS_LINEAR)
