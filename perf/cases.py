"""Timed cases of the NVFP4 hot path, each through the entry point a user's program calls.

    linear    ops.nvfp4_linear               activation quantizer + GEMM of a dense layer (prefill and decode)
    quantize  ops.scaled_fp4_quant           the stand-alone activation quantizer
    decode    sparse_fp4_v7.FusedSparseMoE   one 2:4-sparse MoE layer for a decode batch
    prefill   grouped_moe.nvfp4_moe_prefill  one dense-NVFP4 MoE layer for a block of prompt tokens
    router    router.moe_router              gate projection + softmax + top-k
    convert   sparse_fp4_v7.convert_weight_batch_to_v7   a layer's expert weights to the 2:4 form when a model is loaded

`listed()` holds the sizes that are looked at one by one, `draw()` gives further ones of the same ranges.  Inputs are
seeded synthetic tensors of the benchmark's distributions: activations N(0,1), weights N(0,0.02)."""
import math

import torch

from dgx_vllm_b200.grouped_moe import nvfp4_moe_alphas, nvfp4_moe_prefill
from dgx_vllm_b200.ops import nvfp4_linear, scaled_fp4_quant
from dgx_vllm_b200.router import moe_router
from dgx_vllm_b200.sparse_fp4_v7 import FusedSparseMoE, convert_weight_batch_to_v7

CODE_MAX = 6.0 * 448.0        # largest E2M1 value times the largest E4M3 block scale
DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16}
HIDDEN = (1024, 1536, 2048, 3072, 4096)
INTER = (256, 384, 512, 768, 1024)
EXPERTS = (64, 128, 256, 512)

# What no drawn case exceeds: the largest listed one of its kind.
MAX_LINEAR = 4096 * 14336 * 4096
MAX_WEIGHT = 14336 * 4096
MAX_QUANT = 16384 * 4096
MAX_EXPERTS = 512 * 2048 * 512
MAX_PREFILL = 8192 * 10 * 2048 * 512
MAX_CONVERT = 512 * 1024 * 2048


def listed():
    return [
        # one small projection of a few decoding sequences: launches and host time are all there is
        dict(name="linear_m8", kind="linear", M=8, N=512, K=2048, dtype="bf16"),
        # a wide MLP projection for a decode batch: the weight is read once for few tokens
        dict(name="linear_m128", kind="linear", M=128, N=14336, K=4096, dtype="bf16"),
        # the same projection for a full prompt: bound by the tensor cores
        dict(name="linear_m4096", kind="linear", M=4096, N=14336, K=4096, dtype="bf16"),
        # a prompt of no round length through a layer of no round width, f16 model
        dict(name="linear_ragged", kind="linear", M=777, N=3000, K=4160, dtype="f16"),
        # quantizing a long prompt's activations for a layer (also how a weight is quantized)
        dict(name="quantize_16384", kind="quantize", M=16384, K=4096, dtype="bf16", swizzled=True),
        # one user decoding: ten experts of 512 for one token
        dict(name="decode_b1", kind="decode", M=1, E=512, H=2048, I=512, topk=10, dtype="bf16"),
        # the usual decode batch: about half of the experts are read for a few tokens each
        dict(name="decode_b32", kind="decode", M=32, E=512, H=2048, I=512, topk=10, dtype="bf16"),
        # the largest decode batch: nearly every expert is read
        dict(name="decode_b128", kind="decode", M=128, E=512, H=2048, I=512, topk=10, dtype="bf16"),
        # a full prefill block: a few popular experts get thousands of rows, most get tens
        dict(name="prefill_8192", kind="prefill", M=8192, E=512, H=2048, I=512, topk=10, skewed=True, dtype="bf16"),
        # a short prompt of no round length: most experts get a handful of rows
        dict(name="prefill_611", kind="prefill", M=611, E=512, H=2048, I=512, topk=10, skewed=True, dtype="bf16"),
        # routing a decode batch
        dict(name="router_b32", kind="router", M=32, E=512, H=2048, topk=10, renormalize=True, dtype="bf16"),
        # loading a checkpoint: the gate_up weights of one layer's 512 experts
        dict(name="convert_512", kind="convert", E=512, N=1024, K=2048),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _moe_shape(rng):
    """Hidden size, intermediate size and expert count whose weights are no larger than the listed layer's."""
    while True:
        H, I, E = rng.choice(HIDDEN), rng.choice(INTER), rng.choice(EXPERTS)
        if E * H * I <= MAX_EXPERTS:
            return H, I, E


def draw(rng):
    """One more case of the listed ranges: token counts, widths and depths spread over their logarithm, odd ones among them."""
    kind = rng.choice(("linear", "linear", "quantize", "decode", "decode", "prefill", "router", "convert"))
    dtype = rng.choice(("bf16", "bf16", "f16"))
    if kind == "linear":
        while True:
            M, N, K = _log(rng, 1, 4096), 8 * _log(rng, 64, 2048), 64 * _log(rng, 8, 128)
            if N * K <= MAX_WEIGHT and M * N * K <= MAX_LINEAR:
                return dict(kind=kind, M=M, N=N, K=K, dtype=dtype)
    if kind == "quantize":
        while True:
            M, K = _log(rng, 1, 16384), 16 * _log(rng, 32, 512)
            if M * K <= MAX_QUANT:
                return dict(kind=kind, M=M, K=K, dtype=dtype, swizzled=rng.random() < 0.75)
    if kind == "decode":
        H, I, E = _moe_shape(rng)
        return dict(kind=kind, M=_log(rng, 1, 128), E=E, H=H, I=I, topk=rng.choice((4, 8, 10)), dtype=dtype)
    if kind == "prefill":
        while True:
            (H, I, E), M, topk = _moe_shape(rng), _log(rng, 64, 8192), rng.choice((4, 8, 10))
            if M * topk * H * I <= MAX_PREFILL:
                return dict(kind=kind, M=M, E=E, H=H, I=I, topk=topk, skewed=rng.random() < 0.5, dtype=dtype)
    if kind == "router":
        return dict(kind=kind, M=_log(rng, 1, 8192), E=rng.choice(EXPERTS), H=rng.choice(HIDDEN), topk=rng.choice((4, 8, 10)),
                    renormalize=rng.random() < 0.75, dtype=dtype)
    while True:
        (H, I, E), down = _moe_shape(rng), rng.random() < 0.5
        N, K = (H, I) if down else (2 * I, H)
        if E * N * K <= MAX_CONVERT:
            return dict(kind=kind, E=E, N=N, K=K)


def _gs(amax):
    return torch.full((1,), CODE_MAX / amax, dtype=torch.float32, device="cuda")


def _weights(rows, K, gen, swizzled):
    """[rows, K] N(0, 0.02) weights quantized with one global scale -> (codes, block scales, global scale)."""
    gs = _gs(0.02 * 6.5)
    w = torch.randn(rows, K, generator=gen, device="cuda", dtype=torch.bfloat16).mul_(0.02)
    codes, sf = scaled_fp4_quant(w, gs, swizzled)
    return codes, sf, gs


def _expert_weights(E, N, K, gen, swizzled):
    """Codes [E,N,K/2], block scales and a global scale per expert; made in parts so that the 16-bit weights stay small."""
    step = max(1, min(E, (1 << 28) // (N * K)))
    codes, sfs = [], []
    for e in range(0, E, step):
        c, s, gs = _weights(min(step, E - e) * N, K, gen, swizzled)
        codes.append(c)
        sfs.append(s.view(torch.uint8))
    spread = 0.9 + 0.2 * torch.rand(E, generator=gen, device="cuda")      # the experts' largest weights differ
    codes = torch.cat(codes).view(E, N, K // 2)
    sf = torch.cat(sfs)
    return codes, sf.view(E, -1) if swizzled else sf.view(E, N, K // 16), gs * spread


def _routing(M, E, topk, gen, skewed):
    """Top-k routing: softmax of N(0,1) logits, or experts drawn with a Zipf(1.1) popularity; weights add up to one."""
    if skewed:
        rank = torch.randperm(E, generator=gen, device="cuda").float() + 1.0
        u = torch.rand(M, E, generator=gen, device="cuda").clamp_min(1e-20)
        ids = (-1.1 * torch.log(rank) - torch.log(-torch.log(u))).topk(topk, dim=-1).indices
        w = torch.softmax(torch.randn(M, topk, generator=gen, device="cuda"), dim=-1)
    else:
        w, ids = torch.softmax(torch.randn(M, E, generator=gen, device="cuda"), dim=-1).topk(topk, dim=-1)
        w = w / w.sum(-1, keepdim=True)
    return w.float().contiguous(), ids.to(torch.int32).contiguous()


def prepare(case, seed):
    """What the program holds before the call: its inputs, and the weights and handles it has laid out once."""
    c = case
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = c["kind"]
    if kind == "convert":
        codes, sf, gs = _expert_weights(c["E"], c["N"], c["K"], gen, False)
        return dict(kind=kind, args=(codes, sf.view(torch.float8_e4m3fn), 1.0 / gs))
    dtype = DTYPES[c["dtype"]]
    if kind == "quantize":
        x = torch.randn(c["M"], c["K"], generator=gen, device="cuda", dtype=dtype)
        return dict(kind=kind, args=(x, _gs(6.5), c["swizzled"]))
    if kind == "linear":
        codes, sf, gw = _weights(c["N"], c["K"], gen, True)
        x = torch.randn(c["M"], c["K"], generator=gen, device="cuda", dtype=dtype)
        gx = _gs(6.5)
        return dict(kind=kind, args=(x, gx, codes, sf, (1.0 / (gx * gw)).float()))
    if kind == "router":
        gate = torch.randn(c["E"], c["H"], generator=gen, device="cuda", dtype=dtype).mul_(c["H"] ** -0.5)
        x = torch.randn(c["M"], c["H"], generator=gen, device="cuda", dtype=dtype)
        return dict(kind=kind, args=(x, gate, c["topk"], c["renormalize"]))
    E, H, I = c["E"], c["H"], c["I"]
    x = torch.randn(c["M"], H, generator=gen, device="cuda", dtype=dtype)
    w, ids = _routing(c["M"], E, c["topk"], gen, c.get("skewed", False))
    if kind == "decode":
        bound = []
        for N, K in ((2 * I, H), (H, I)):
            codes, sf, gs = _expert_weights(E, N, K, gen, False)
            bound += convert_weight_batch_to_v7(codes, sf, 1.0 / gs)
        return dict(kind=kind, layer=FusedSparseMoE(*bound, I), args=(x, w, ids))
    w13, sf13, gs13 = _expert_weights(E, 2 * I, H, gen, True)
    w2, sf2, gs2 = _expert_weights(E, H, I, gen, True)
    a1 = _gs(6.5).expand(E).contiguous()
    a2 = _gs(12.0).expand(E).contiguous()
    return dict(kind=kind, args=(x, w, ids, w13, sf13, gs13, w2, sf2, gs2, a1, a2),
                alphas=nvfp4_moe_alphas(gs13, gs2, a1, a2))


def run(state):
    kind, args = state["kind"], state["args"]
    if kind == "linear":
        return nvfp4_linear(*args)
    if kind == "quantize":
        return scaled_fp4_quant(*args)
    if kind == "decode":
        return state["layer"](*args)
    if kind == "prefill":
        return nvfp4_moe_prefill(*args, alphas=state["alphas"])
    if kind == "router":
        return moe_router(*args)
    return convert_weight_batch_to_v7(*args)


def _experts_read(c):
    """Expected number of experts that get at least one token."""
    if c.get("skewed"):
        p = [(i + 1) ** -1.1 for i in range(c["E"])]
        s = sum(p)
        return sum(1.0 - (1.0 - q / s) ** (c["M"] * c["topk"]) for q in p)
    return c["E"] * (1.0 - (1.0 - c["topk"] / c["E"]) ** c["M"])


def work(case):
    """Bytes: each input read once, each output written once (an expert's weights only if a token uses it).  Operations:
    multiplications and additions of the products, of the kept half of the weights where they are 2:4 sparse."""
    c = case
    kind = c["kind"]
    if kind == "linear":
        M, N, K = c["M"], c["N"], c["K"]
        return {"bytes": 2 * M * K + N * K * 9 / 16 + 2 * M * N, "flops": 2 * M * N * K}
    if kind == "quantize":
        return {"bytes": c["M"] * c["K"] * (2 + 9 / 16), "flops": 0}
    if kind == "convert":
        # codes and scales in; kept codes, their positions and scales out
        return {"bytes": c["E"] * c["N"] * c["K"] * (1 / 2 + 1 / 16 + 1 / 4 + 1 / 8 + 1 / 16), "flops": 0}
    M, E, H, topk = c["M"], c["E"], c["H"], c["topk"]
    if kind == "router":
        return {"bytes": 2 * M * H + 2 * E * H + 8 * M * topk, "flops": 2 * M * E * H}
    weights = 3 * H * c["I"]
    per_weight, flops = (7 / 16, 1) if kind == "decode" else (9 / 16, 2)
    return {"bytes": _experts_read(c) * weights * per_weight + 4 * M * H + 8 * M * topk, "flops": flops * M * topk * weights}


def tolerance(case):
    kind = case["kind"]
    if kind in ("quantize", "convert"):
        return "exact"
    if kind == "router":
        return {"rel": 1e-4, "max": 1e-2, "differ": 2e-3}      # f32 sums; logits closer than their rounding may swap places
    if kind == "prefill":
        return {"rel": 1e-2}       # 16-bit output, and a last-bit difference before the second quantizer moves a 4-bit code
    return {"rel": 5e-3}           # one rounding to 16 bits of f32 sums (decode: the products between the projections are f16)
