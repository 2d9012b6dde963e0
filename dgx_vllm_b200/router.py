"""MoE router on the GPU: gate projection + softmax + top-k + renormalisation in one or two small kernels, producing the
(topk_weights f32, topk_ids i32) pair the fused MoE ops take.  The reference leaves this step to vLLM; its benches
restate it in torch (sparse_fp4_kernel/bench_moe_layer_e2e.py:230-236), which is what the parity test compares with."""
from __future__ import annotations

import torch

from . import _lib
from ._torch_util import WS_ROUTER, status_word


def moe_router(hidden_states: torch.Tensor, gate_weight: torch.Tensor, topk: int, renormalize: bool = True):
    """hidden_states [M,H], gate_weight [E,H] (both bf16 or both f16) -> (topk_weights [M,topk] f32, topk_ids [M,topk] i32).
    Weights are softmax probabilities of the selected experts, divided by their sum when renormalize is set."""
    return _lib.host().moe_router(hidden_states, gate_weight, topk, renormalize)


def last_router_status(device=None) -> int:
    """Status word of the most recent moe_router on the current stream of `device`: 0, or the code of a bounded wait that ran
    out in the projection of many tokens (that call's weights and ids are then not valid).  Synchronises."""
    return status_word(device, WS_ROUTER)
