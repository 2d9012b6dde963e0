"""The native host path among several Python threads: a call that waits for its stream's queue leaves the interpreter to the
others, and calls of two threads on one stream keep their steps and scratch apart."""
import threading
import time

import pytest
import torch

import synth
from util import gpu_quantize_fn

pytestmark = pytest.mark.gpu


def _gs(v):
    return torch.full((1,), v, device="cuda")


def _calls():
    """One small call of every entry of the native host path."""
    from dgx_vllm_b200 import cutlass_scaled_fp4_mm, scaled_fp4_quant, sparse_fp4_v7 as sp7
    from dgx_vllm_b200.grouped_moe import nvfp4_moe_alphas, nvfp4_moe_prefill
    from dgx_vllm_b200.ops import nvfp4_linear
    from dgx_vllm_b200.router import moe_router
    E, H, I, M, topk = 4, 256, 128, 4, 2
    x, gs = synth.make_hidden(M, H, 0, "cuda"), _gs(400.0)
    wc, ws = scaled_fp4_quant(synth.make_hidden(128, H, 1, "cuda"), gs)
    xc, xs = scaled_fp4_quant(x, gs)
    alpha = 1.0 / (gs * gs)
    tw, ids = synth.make_routing(M, E, topk, 2, "cuda")
    keys = ("comp_T", "meta_T", "scale_T", "g_scales")
    w13, w2 = (synth.make_sparse_experts(E, n, k, 3, "cuda", gpu_quantize_fn) for n, k in ((2 * I, H), (H, I)))
    layer = sp7.FusedSparseMoE(*[w13[k] for k in keys], *[w2[k] for k in keys], I)

    def dense(N, K):
        c, s = scaled_fp4_quant(synth.make_hidden(E * N, K, 4, "cuda"), gs)
        return c.view(E, N, K // 2), s.view(torch.uint8).view(E, -1), gs.expand(E).contiguous()
    d13, d2, a = dense(2 * I, H), dense(H, I), gs.expand(E).contiguous()
    alphas = nvfp4_moe_alphas(d13[2], d2[2], a, a)
    return {
        "quant": lambda: scaled_fp4_quant(x, gs),
        "mm": lambda: cutlass_scaled_fp4_mm(xc, wc, xs, ws, alpha, torch.bfloat16),
        "linear": lambda: nvfp4_linear(x, gs, wc, ws, alpha),
        "router": lambda: moe_router(x, x.repeat(2, 1), topk),
        "decode": lambda: layer(x, tw, ids),
        "prefill": lambda: nvfp4_moe_prefill(x, tw, ids, *d13, *d2, a, a, alphas=alphas),
    }


@pytest.mark.parametrize("name", ["quant", "mm", "linear", "router", "decode", "prefill"])
def test_a_full_queue_does_not_stop_other_threads(name):
    call = _calls()[name]
    call()
    torch.cuda.synchronize()
    ticks, stop = [], threading.Event()

    def tick():
        while not stop.is_set():
            ticks.append(time.perf_counter())
            time.sleep(0.001)

    t = threading.Thread(target=tick)
    t.start()
    try:
        torch.cuda._sleep(1_500_000_000)              # about 0.8 s of a kernel in front of the queue
        t0 = time.perf_counter()
        for _ in range(2500):
            call()
        waited = time.perf_counter() - t0
    finally:
        stop.set()
        t.join()
        torch.cuda.synchronize()
    assert waited > 0.4, "the queue never filled"
    assert max(b - a for a, b in zip(ticks, ticks[1:])) < 0.5 * waited        # the GIL held: as long as the wait


def test_two_threads_on_one_stream_keep_their_calls_apart():
    from dgx_vllm_b200 import scaled_fp4_quant
    from dgx_vllm_b200.ops import nvfp4_linear
    K, N, gs = 1024, 256, _gs(400.0)
    wc, ws = scaled_fp4_quant(synth.make_hidden(N, K, 9, "cuda"), gs)
    alpha = 1.0 / (gs * gs)
    # the scratch of a call grows with its rows: both threads make the stream's scratch grow, in steps
    xs = [[synth.make_hidden(m, K, i, "cuda") for m in (40 + i, 900 + i, 2100 + i, 4200 + i)] for i in range(2)]
    want = [[nvfp4_linear(x, gs, wc, ws, alpha) for x in part] for part in xs]
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    wrong, errors = [0, 0], []

    def work(i):
        try:
            with torch.cuda.stream(stream):
                for j in range(4):
                    got = [nvfp4_linear(xs[i][j], gs, wc, ws, alpha) for _ in range(60)]
                    wrong[i] += sum(not torch.equal(g, want[i][j]) for g in got)
        except Exception as e:                        # shown by the assertion below
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors and wrong == [0, 0]
