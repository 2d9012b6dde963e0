"""GPU parity at the sizes where a kernel's tiling can go wrong: tile edges, remainders, smallest and largest of a range."""
import numpy as np
import pytest
import torch

import oracle
from util import to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,N,K,G", [
    (2, 128, 256, 16),       # one whole tile
    (1, 1, 8, 1),            # smallest
    (2, 129, 264, 33),       # one past a tile both ways; rows of no whole 16-byte chunk, byte stores
    (2, 132, 288, 18),       # width a multiple of four only, whole chunks of codes but not of scales
    (2, 144, 512, 32),       # a tile and one 16-column group
    (3, 36, 1024, 64),       # several tiles along k, columns past the row end
])
def test_convert_2of4_tile_edges(E, N, K, G):
    from dgx_vllm_b200 import sparse_fp4_v7 as sp7
    rng = np.random.default_rng(N + K)
    codes = rng.integers(0, 256, (E, N, K // 2), dtype=np.uint8)
    sf = rng.integers(0, 256, (E, N, G), dtype=np.uint8)
    comp, meta, scale, _ = sp7.convert_weight_batch_to_v7(torch.from_numpy(codes), torch.from_numpy(sf), torch.ones(E))
    for e in range(E):
        oc, om = oracle.sparse_2of4_pack(codes[e])
        np.testing.assert_array_equal(to_np(comp[e]), oc)
        np.testing.assert_array_equal(to_np(meta[e]), om)
        np.testing.assert_array_equal(to_np(scale[e]), sf[e].T)


@pytest.mark.parametrize("M,H,E,topk,dtype,renorm", [
    (1, 8, 1, 1, torch.bfloat16, True),               # smallest: one 16-byte piece of K, one expert
    (9, 1000, 40, 5, torch.float16, True),            # one past eight tokens, K no multiple of 64, experts past a block of 16
    (64, 512, 64, 8, torch.bfloat16, True),           # last size of the small-batch kernel
    (65, 2048, 1024, 32, torch.bfloat16, False),      # first of the tile kernel, largest E and topk
    (257, 520, 136, 8, torch.float16, True),          # tokens, experts and K past their tiles
    (1024, 2048, 512, 10, torch.bfloat16, True),      # several K-slices
    (4864, 1024, 512, 10, torch.bfloat16, False),     # 256-wide expert tiles
    (4865, 256, 290, 4, torch.float16, True),         # ... past their end, E no multiple of four
    (17, 4096, 128, 8, torch.bfloat16, False),        # clusters of eight: one tile of experts to a block, sixteen slices of K
    (31, 72, 129, 4, torch.float16, True),            # clusters of sixteen, most blocks without experts, less K than slices
    (56, 2048, 512, 10, torch.bfloat16, False),       # ... as many as run at once
    (64, 1024, 500, 10, torch.float16, False),        # ... one more: clusters of eight again, four tiles to a block
    (16, 1000, 1023, 32, torch.bfloat16, True),       # more than 512 experts
    (3, 12800, 600, 4, torch.bfloat16, True),         # ... with a gate for K-slices: eight tokens a block
    (3, 12800, 1000, 4, torch.bfloat16, True),        # ... and for the tile kernel
    (8, 1544, 1, 1, torch.float16, True),             # K-slices: one expert, the last of four slices with little to do
    (7, 3080, 33, 5, torch.bfloat16, False),          # ... experts past a block
    (16, 2568, 64, 8, torch.float16, True),           # ... sixteen tokens a block
    (9, 12800, 511, 10, torch.bfloat16, True),        # ... fewer tokens than that
    (17, 1032, 640, 10, torch.bfloat16, True),        # ... thirty-two
    (32, 4608, 1024, 32, torch.float16, False),       # ... the largest
    (33, 1024, 640, 10, torch.bfloat16, True),        # one more: tiles
])
def test_router_kernel_edges(M, H, E, topk, dtype, renorm):
    from dgx_vllm_b200.router import moe_router
    g = torch.Generator(device="cuda").manual_seed(M + E)
    wide = torch.randn(M, H + 8, generator=g, device="cuda").to(dtype)
    hidden = wide[:, :H]                              # strided rows
    gate = (torch.randn(E, H, generator=g, device="cuda") / H ** 0.5).to(dtype)
    results = [moe_router(hidden, gate, topk, renormalize=renorm)]
    graph = torch.cuda.CUDAGraph()                    # takes the K-slices at more sizes
    with torch.cuda.graph(graph):
        results.append(moe_router(hidden, gate, topk, renormalize=renorm))
    graph.replay()
    torch.cuda.synchronize()
    logits = hidden.double() @ gate.double().t()
    w, ref_ids = torch.softmax(logits, dim=-1).topk(topk, dim=-1)
    if renorm:
        w = w / w.sum(-1, keepdim=True)
    srt = torch.cat((logits, torch.full((M, 1), -1e9, device="cuda", dtype=torch.double)), 1).sort(dim=-1, descending=True).values
    clear = (srt[:, :topk] - srt[:, 1:topk + 1]).min(dim=-1).values > 2e-5
    assert clear.float().mean() > 0.8
    for tw, ids in results:
        assert torch.equal(ids[clear].long(), ref_ids[clear])
        assert ((tw[clear].double() - w[clear]).abs() / w[clear]).max() < 1e-4


@pytest.mark.parametrize("M,H,E,launches,captured", [
    (8, 1536, 32, 1, 1), (8, 2048, 32, 1, 2), (8, 10240, 32, 1, 2), (8, 10248, 32, 2, 2), (16, 2560, 64, 1, 1), (16, 4096, 64, 1, 2),
    (8, 6144, 128, 1, 1), (8, 7168, 128, 1, 2), (16, 12800, 128, 2, 2), (17, 12800, 128, 1, 1), (8, 6144, 512, 1, 1), (8, 9216, 512, 2, 2),
    (16, 7168, 512, 1, 1), (32, 9216, 512, 1, 1), (4, 3072, 1000, 1, 1), (4, 4096, 1000, 2, 2), (17, 2048, 1000, 2, 2),
])
def test_router_path(M, H, E, launches, captured):
    # clusters in one launch, or two launches that have every SM read its share of a large gate: the second launch costs little in a graph only
    from dgx_vllm_b200 import _lib
    from dgx_vllm_b200.router import moe_router
    x, gate = torch.zeros(M, H, device="cuda", dtype=torch.bfloat16), torch.zeros(E, H, device="cuda", dtype=torch.bfloat16)
    n0 = _lib.lib().b200fp4_launch_count()
    results = [moe_router(x, gate, 8)]
    assert _lib.lib().b200fp4_launch_count() == n0 + launches
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        results.append(moe_router(x, gate, 8))
    assert _lib.lib().b200fp4_launch_count() == n0 + launches + captured
    graph.replay()
    torch.cuda.synchronize()
    for tw, ids in results:
        assert torch.equal(ids, torch.arange(8, device="cuda", dtype=torch.int32).expand(M, 8)) and bool((tw == 0.125).all())


@pytest.mark.parametrize("E", [1, 32, 128, 512, 513, 1000])
def test_router_workspace_of_a_larger_batch(E):
    # a program that sizes its workspace for its largest decode batch may call with fewer tokens, whichever path these take
    from dgx_vllm_b200 import _lib
    from dgx_vllm_b200.router import moe_router
    L, most, topk = _lib.lib(), 64, min(E, 8)
    sizes = [L.b200fp4_moe_router_workspace_bytes(m, E) for m in range(1, 129)]
    assert sizes == sorted(sizes)
    nbytes, st = sizes[most - 1], torch.cuda.current_stream().cuda_stream
    for M, H in [(8, 1536), (8, 12800), (16, 12800), (32, 4096), (64, 2048)]:
        g = torch.Generator(device="cuda").manual_seed(M + H)
        x, gate = (torch.randn(n, H, generator=g, device="cuda").mul_(H ** -0.25).bfloat16() for n in (M, E))
        ws = torch.full((nbytes + 256,), 77, dtype=torch.uint8, device="cuda")
        tw, ids = torch.empty(M, topk, device="cuda"), torch.empty(M, topk, dtype=torch.int32, device="cuda")
        _lib.check(L.b200fp4_moe_router(x.data_ptr(), H, _lib.BF16, gate.data_ptr(), M, H, E, topk, 1, tw.data_ptr(), ids.data_ptr(),
                                        ws.data_ptr(), nbytes, st), "router")
        want = moe_router(x, gate, topk)
        assert torch.equal(tw, want[0]) and torch.equal(ids, want[1])
        assert bool((ws[nbytes:] == 77).all())


@pytest.mark.parametrize("M,K", [(1, 16), (31, 48), (33, 512), (97, 528), (129, 80), (200, 2064)])
@pytest.mark.parametrize("swizzled", [True, False])
@pytest.mark.parametrize("offset", [0, 8])            # elements: rows on 32-byte and only on 16-byte boundaries
def test_quantizer_tile_edges(M, K, swizzled, offset):
    from dgx_vllm_b200 import scaled_fp4_quant
    from util import bf16_bits
    g = torch.Generator().manual_seed(M * K)
    wide = torch.randn(M, K + 16, generator=g).to(torch.bfloat16)
    wide[0, offset:offset + 16] = 0.0                 # a block of zeros
    x = wide[:, offset:offset + K]
    gs = torch.tensor([448.0 * 6.0 / 4.0])
    codes, sf = scaled_fp4_quant(wide.cuda()[:, offset:offset + K], gs.cuda(), swizzled)
    ref_codes, ref_sf = oracle.quantize_bf16(bf16_bits(x.contiguous()), float(gs[0]))
    np.testing.assert_array_equal(to_np(codes), ref_codes)
    got = to_np(sf)
    if swizzled:                                      # padding included: zeros past M and past K / 16
        ref_sf = np.asarray(oracle.sf_linear_to_swizzled(ref_sf)).reshape(got.shape)
    np.testing.assert_array_equal(got, ref_sf)


@pytest.mark.parametrize("E,H,I,M,topk", [
    (4, 256, 128, 1, 1),          # smallest: one pair and that not local, on the path for few pairs
    (1, 256, 128, 2, 1),          # smallest of the one-launch kernel: one item, K = 128 on the down side; two warps per item, down turns of two
    (8, 512, 512, 3, 4),          # four warps per item
    (16, 256, 256, 32, 8),        # 256 pairs: last size of the small plan; several passes per expert
    (16, 256, 256, 33, 8),        # 264 pairs
    (128, 1024, 768, 25, 10),     # 12 warps, two per item, nine items an SM
    (512, 512, 512, 64, 8),       # ... 17
    (256, 256, 512, 60, 10),      # 16 warps, items of about one round
    (8, 512, 384, 3, 4),          # four warps per item, down slices of three steps
    (8, 1024, 256, 3, 4),         # ... of two
    (128, 512, 384, 40, 4),       # 12 warps, two per item, down turns of three
    (256, 512, 384, 64, 4),       # eight warps, one per item, down turns of four
    (256, 512, 512, 25, 8),       # ... of eight
    (8, 384, 128, 200, 4),        # 16 warps, one per item: K no multiple of 256, many pairs per expert
    (64, 512, 1024, 256, 10),     # 16 warps, many items of several passes per expert
])
def test_fused_moe_block_shapes(E, H, I, M, topk):
    import synth
    from dgx_vllm_b200 import _lib, sparse_fp4_v7 as sp7
    from util import expert_fetch, gpu_quantize_fn, rel_err
    keys = ("comp_T", "meta_T", "scale_T", "g_scales")
    w13 = synth.make_sparse_experts(E, 2 * I, H, 1, "cuda", gpu_quantize_fn)
    w2 = synth.make_sparse_experts(E, H, I, 2, "cuda", gpu_quantize_fn)
    tw, ids = synth.make_routing(M, E, topk, 3, "cuda")
    ids[0, 0] = -1                                    # not local
    hidden = synth.make_hidden(M, H, 4, "cuda")
    args = (hidden, tw, ids, None, *[w13[k] for k in keys], *[w2[k] for k in keys], I, False)
    n0 = _lib.lib().b200fp4_launch_count()
    out = sp7.fused_sparse_moe_v7(*args)
    assert _lib.lib().b200fp4_launch_count() == n0 + (3 if 2 * M * topk > E else 2)      # few pairs have no plan
    again = sp7.fused_sparse_moe_v7(*args)
    assert sp7.last_moe_status() == 0
    assert torch.equal(out, again)
    ref = oracle.fused_sparse_moe_by_expert(hidden.float().cpu().numpy(), tw.cpu().numpy(), ids.cpu().numpy(), expert_fetch(w13, w2), I)
    assert rel_err(to_np(out), ref) < 1e-2


@pytest.mark.parametrize("M,N,K", [
    (1, 8, 2048),             # few tokens: K over eight CTAs, one row and less than a 32-column piece
    (33, 136, 2112),          # ... ragged everywhere, last k-stage short
    (129, 1000, 4096),        # split of K over four CTAs, two row tiles
    (5, 5000, 1024),          # few tokens, over three
    (200, 4096, 1088),        # five stages: no split
    (70, 136, 2112),          # split over four, ragged everywhere, last k-stage short
    (130, 2304, 4160),        # ... over two
    (8, 264, 768),            # three stages: no split
    (385, 6000, 1024),        # wide tiles, ragged
    (520, 7000, 2048),        # pairs of CTAs, ragged
])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_dense_gemm_tile_choice(M, N, K, dtype):
    from dgx_vllm_b200 import cutlass_scaled_fp4_mm, scaled_fp4_quant
    from dgx_vllm_b200.ops import last_gemm_status
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(N, K, generator=g, device="cuda").mul_(0.02).to(torch.bfloat16)
    gx, gw = torch.full((1,), 2688 / 6.5, device="cuda"), torch.full((1,), 2688 / 0.13, device="cuda")
    (xc, xs), (wc, ws) = scaled_fp4_quant(x, gx), scaled_fp4_quant(w, gw)
    alpha = 1.0 / (gx * gw)
    guard = torch.full((M * N + 64,), 7.0, dtype=dtype, device="cuda")       # nothing past the result is touched
    out = guard[:M * N].view(M, N)
    cutlass_scaled_fp4_mm(xc, wc, xs, ws, alpha, dtype, out=out)
    assert last_gemm_status() == 0
    assert bool((guard[M * N:] == 7.0).all())

    def deq(codes, sf, gs, rows):
        lin = oracle.sf_swizzled_to_linear(to_np(sf).reshape(-1), rows, K // 16)
        return torch.from_numpy(oracle.dequantize(to_np(codes), lin, float(gs[0]))).cuda().double()
    ref = (deq(xc, xs, gx, M) @ deq(wc, ws, gw, N).t()).float()
    assert ((out.float() - ref).abs().max() / ref.abs().max()).item() < 5e-3


def _linear_operands(M, N, K, seed):
    from dgx_vllm_b200 import scaled_fp4_quant
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(N, K, generator=g, device="cuda").mul_(0.02).to(torch.bfloat16)
    gx, gw = torch.full((1,), 2688 / 6.5, device="cuda"), torch.full((1,), 2688 / 0.13, device="cuda")
    return x, gx, *scaled_fp4_quant(w, gw), 1.0 / (gx * gw)


@pytest.mark.parametrize("M,N,K", [
    (8, 512, 2048),           # few tokens: one kernel, K over eight CTAs
    (33, 136, 2112),          # ... ragged, nine stages on eight CTAs, the last one short
    (129, 1000, 4096),        # quantizer and GEMM, K split over four CTAs: every CTA requests its own first stages early
    (5, 5000, 1024),          # few tokens, over three
    (8, 264, 64),             # ... a single short stage
    (128, 14336, 1024),       # narrow tiles, fewer stages than the ring holds
    (385, 6000, 1088),        # wide tiles; the columns of the second scale tile lie past N
    (70, 136, 2112),          # more tokens than the few-token kernel takes: split over four, nine stages, the last one short
    (130, 2304, 4160),        # ... over two, 36 tiles of 17 stages
    (72, 264, 64),            # ... a single short stage
])
def test_linear_early_weights(M, N, K):
    from dgx_vllm_b200 import cutlass_scaled_fp4_mm, scaled_fp4_quant
    from dgx_vllm_b200.ops import last_gemm_status, nvfp4_linear
    x, gx, wc, ws, alpha = _linear_operands(M, N, K, M + K)
    out = nvfp4_linear(x, gx, wc, ws, alpha)
    assert last_gemm_status() == 0
    xc, xs = scaled_fp4_quant(x, gx)
    assert torch.equal(out, cutlass_scaled_fp4_mm(xc, wc, xs, ws, alpha, torch.bfloat16))


@pytest.mark.parametrize("M", [8, 128, 300])
@pytest.mark.parametrize("last", ["codes", "scales", "quantizer"])
def test_linear_reads_weights_the_kernel_before_it_wrote(M, last):
    # the GEMM requests weights before it waits for the quantizer; the quantizer lets it start only after whatever wrote them
    from dgx_vllm_b200 import scaled_fp4_quant
    from dgx_vllm_b200.ops import nvfp4_linear
    N, K, rounds = 4096, 4096, 12
    sets = [_linear_operands(M, N, K, s) for s in range(2)]
    x, gx, alpha = sets[0][0], sets[0][1], sets[0][4]
    want = [nvfp4_linear(x, gx, s[2], s[3], alpha) for s in sets]
    assert not torch.equal(*want)
    dense = [torch.randn(N, K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(s)).mul_(0.02).bfloat16() for s in (5, 6)]
    gw = torch.full((1,), 2688 / 0.13, device="cuda")
    if last == "quantizer":
        want = [nvfp4_linear(x, gx, *scaled_fp4_quant(d, gw), alpha) for d in dense]
    codes, sf = torch.empty_like(sets[0][2]), torch.empty_like(sets[0][3])
    torch.cuda.synchronize()
    got = []
    torch.cuda._sleep(4_000_000)                      # everything below is queued before the first of it runs
    for i in range(rounds):
        if last == "quantizer":
            codes, sf = scaled_fp4_quant(dense[i % 2], gw)
        else:
            copy = [lambda: torch.bitwise_or(sets[i % 2][2], 0, out=codes),
                    lambda: torch.bitwise_or(sets[i % 2][3].view(torch.uint8), 0, out=sf.view(torch.uint8))]
            for c in copy if last == "scales" else copy[::-1]:
                c()
        got.append(nvfp4_linear(x, gx, codes, sf, alpha))
    torch.cuda.synchronize()
    assert all(torch.equal(g, want[i % 2]) for i, g in enumerate(got))


@pytest.mark.parametrize("M,E,topk,H,I,dtype", [
    (1, 4, 1, 64, 128, torch.bfloat16),          # one row, less than one 256-wide stage of k
    (37, 4, 3, 320, 128, torch.float16),         # a tail stage of one k-block
    (200, 2, 2, 704, 256, torch.bfloat16),       # tail of three k-blocks, several row tiles per expert
    (65, 8, 5, 1024, 384, torch.bfloat16),       # a batch of four slots and one more
    (33, 16, 16, 4160, 128, torch.float16),      # a row longer than a block of threads takes at once
    (16384, 8, 8, 64, 128, torch.bfloat16),      # 131,072 pairs: the most that one launch routes
    (16385, 8, 8, 64, 128, torch.bfloat16),      # ... more: grid-wide routing steps, the tile list made by the first GEMM
])
def test_prefill_layer_equals_its_steps(M, E, topk, H, I, dtype):
    from dgx_vllm_b200 import grouped_moe as gm
    from dgx_vllm_b200.ops import last_gemm_status, scaled_fp4_quant
    g = torch.Generator(device="cuda").manual_seed(M + H)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    hidden = rnd(M, H).to(dtype)
    tw, ids = torch.softmax(rnd(M, E), -1).topk(topk, -1)
    tw, ids = tw.contiguous(), ids.int().contiguous()

    def weights(N, K):
        gs = torch.full((1,), 6.0 * 448.0 / 0.13, device="cuda")
        c, s = zip(*[scaled_fp4_quant((0.02 * rnd(N, K)).to(dtype), gs, True) for _ in range(E)])
        return torch.stack(c), torch.stack([v.view(torch.uint8) for v in s]).view(E, -1), gs.expand(E).contiguous()

    w13, w2 = weights(2 * I, H), weights(H, I)
    a1, a2 = 400.0 + 50.0 * torch.arange(E, device="cuda").float(), torch.full((E,), 220.0, device="cuda")
    al1, al2 = gm.nvfp4_moe_alphas(w13[2], w2[2], a1, a2)
    out = gm.nvfp4_moe_prefill(hidden, tw, ids, *w13, *w2, a1, a2, alphas=(al1, al2))
    assert last_gemm_status() == 0
    P = M * topk
    eo, a_map, c_map = (torch.empty(n, dtype=torch.int32, device="cuda") for n in (E + 1, P, P))
    bso = gm.get_cutlass_moe_mm_data(ids, eo, None, None, a_map, c_map, E, I, H, pair_indices=True)
    xq, xsf = gm.scatter_scaled_fp4_experts_quant(hidden, c_map, topk, a1, eo, bso, ids, None)
    hq, hsf = gm.cutlass_fp4_moe_mm_silu_and_mul_quant(xq, w13[0], xsf, w13[1], al1, eo, bso, a2, dtype)
    c2 = torch.empty((P, H), dtype=dtype, device="cuda")
    gm.cutlass_fp4_moe_mm(c2, hq, w2[0], hsf, w2[1], al2, None, eo, bso)
    assert torch.equal(out, gm.moe_unpermute_reduce(c2, c_map, tw))
    rows = c2.float()[c_map.long()].view(M, topk, H)
    ref = (rows * tw[..., None]).sum(1)
    assert torch.allclose(out.float(), ref, rtol=1e-2, atol=1e-3 * float(ref.abs().max()))


@pytest.mark.parametrize("M,N,K", [
    (1, 128, 64),              # one tile, one short stage, one column of the narrowest MMA
    (8, 512, 2048),            # a stage to each of the eight CTAs of a cluster
    (9, 130, 2112),            # N past the tile, nine stages on eight CTAs, the last one short
    (16, 14336, 4096),         # K not split, more stages than the ring holds; the most blocks a CTA quantizes
    (17, 1000, 1280),          # five stages on five CTAs
    (31, 2056, 1536),          # clusters of six
    (33, 6400, 768),           # a second word of activation scales
    (39, 392, 5120),           # two or three stages to a CTA, tokens not a multiple of the cluster
    (64, 1024, 4096),          # the most tokens
    (1, 18937, 576),           # as many tiles as SMs
])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_few_token_linear(M, N, K, dtype):
    # the kernel that quantizes its own operand: the same bytes as on codes made before, and the exact product of those codes within
    # one rounding to 16 bits (7 or 10 stored bits: half a unit in the last place is 2^-8 or 2^-11 of the value) and the f32 sum over K
    from dgx_vllm_b200 import _lib, cutlass_scaled_fp4_mm, scaled_fp4_quant
    from dgx_vllm_b200.ops import last_gemm_status, nvfp4_linear
    x, gx, wc, ws, alpha = _linear_operands(M, N, K, M + N)
    x = x.to(dtype)
    n0 = _lib.lib().b200fp4_launch_count()
    out = nvfp4_linear(x, gx, wc, ws, alpha)
    assert _lib.lib().b200fp4_launch_count() == n0 + 1 and last_gemm_status() == 0
    wide = torch.zeros(M, K + 8, dtype=dtype, device="cuda")          # rows that are 16-byte, not 32-byte aligned
    wide[:, :K] = x
    assert torch.equal(nvfp4_linear(wide[:, :K], gx, wc, ws, alpha), out)
    xc, xs = scaled_fp4_quant(x, gx)
    assert torch.equal(cutlass_scaled_fp4_mm(xc, wc, xs, ws, alpha, dtype), out)

    def deq(codes, sf, rows):
        lin = oracle.sf_swizzled_to_linear(to_np(sf.view(torch.uint8)).reshape(-1), rows, K // 16)
        return torch.from_numpy(oracle.dequantize(to_np(codes), lin, 1.0)).cuda().double()

    a, b = deq(xc, xs, M), deq(wc, ws, N)
    ref, size = (a @ b.t()) * alpha.double(), (a.abs() @ b.abs().t()) * alpha.double()
    half_ulp = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    assert bool(((out.double() - ref).abs() <= half_ulp * ref.abs() + 2.0 ** -20 * size + 2.0 ** -24).all())


@pytest.mark.parametrize("gs", [-2688 / 6.5, 0.0, -0.0])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_few_token_linear_any_global_scale(gs, dtype):
    # scale bytes with the sign bit set, and the guard for zero: still the stand-alone quantizer's bytes
    from dgx_vllm_b200 import cutlass_scaled_fp4_mm, scaled_fp4_quant
    from dgx_vllm_b200.ops import nvfp4_linear
    x, _, wc, ws, alpha = _linear_operands(9, 512, 2048, 5)
    x, gx = x.to(dtype), torch.full((1,), gs, device="cuda")
    x[0, :16] = 0.0
    x[1, :16] *= 1e-6                                 # a scale that rounds to zero
    xc, xs = scaled_fp4_quant(x, gx)
    out, want = nvfp4_linear(x, gx, wc, ws, alpha), cutlass_scaled_fp4_mm(xc, wc, xs, ws, alpha, dtype)
    assert torch.equal(out.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("M,E,ranks,topk,launches", [
    (1, 128, 1, 10, 2),           # few pairs: ids and map read by the sum
    (2, 256, 8, 10, 2),           # ... on one of eight expert-parallel ranks, most pairs not local
    (32, 64, 1, 10, 3),           # plan, one launch, sum
    (256, 128, 8, 10, 3),         # ... one local slot of ten on average
    (3, 64, 1, 32, 3),            # every lane of a warp holds a slot
    (3, 64, 4, 40, 3),            # more slots than lanes
])
@pytest.mark.parametrize("written_by", ["router", "copies"])
def test_layer_reads_the_routing_the_kernel_before_it_wrote(M, E, ranks, topk, launches, written_by):
    # the sum looks at its routing before the kernel in front of it ends: ids and weights new for every call, eager and from a graph
    import synth
    from dgx_vllm_b200 import _lib, sparse_fp4_v7 as sp7
    from dgx_vllm_b200.moe_ep import expert_map_for_rank
    from dgx_vllm_b200.router import moe_router
    from util import expert_fetch, gpu_quantize_fn, rel_err
    if written_by == "router" and topk > 32:
        pytest.skip("the router selects up to 32")
    keys, H, I, here = ("comp_T", "meta_T", "scale_T", "g_scales"), 512, 256, E // ranks
    w13 = synth.make_sparse_experts(here, 2 * I, H, 1, "cuda", gpu_quantize_fn)
    w2 = synth.make_sparse_experts(here, H, I, 2, "cuda", gpu_quantize_fn)
    emap = expert_map_for_rank(E, ranks, ranks - 1, "cuda") if ranks > 1 else None
    layer = sp7.FusedSparseMoE(*[w13[k] for k in keys], *[w2[k] for k in keys], I, expert_map=emap)
    gate = torch.randn(E, H, device="cuda", generator=torch.Generator(device="cuda").manual_seed(7)).mul_(H ** -0.5).bfloat16()
    xs = [synth.make_hidden(M, H, 4 + s, "cuda") for s in range(2)]
    routes = [moe_router(x, gate, topk) if topk <= 32 else synth.make_routing(M, E, topk, 8 + s, "cuda") for s, x in enumerate(xs)]
    torch.cuda.synchronize()
    n0 = _lib.lib().b200fp4_launch_count()
    want = [layer(x, *r) for x, r in zip(xs, routes)]
    assert _lib.lib().b200fp4_launch_count() == n0 + 2 * launches
    for x, (tw, ids), got in zip(xs, routes, want):
        local = ids if emap is None else emap[ids.long()]
        ref = oracle.fused_sparse_moe_by_expert(x.float().cpu().numpy(), tw.cpu().numpy(), local.cpu().numpy(), expert_fetch(w13, w2), I)
        assert rel_err(to_np(got), ref) < 1e-2
    tw, ids = torch.zeros_like(routes[0][0]), torch.zeros_like(routes[0][1])

    def step(i):
        if written_by == "router":
            return layer(xs[i % 2], *moe_router(xs[i % 2], gate, topk))
        tw.copy_(routes[i % 2][0])
        ids.copy_(routes[i % 2][1])
        return layer(xs[i % 2], tw, ids)

    torch.cuda.synchronize()
    torch.cuda._sleep(4_000_000)                      # everything below is queued before the first of it runs
    got = [step(i) for i in range(12)]
    torch.cuda.synchronize()
    assert all(torch.equal(g, want[i % 2]) for i, g in enumerate(got))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = [step(i) for i in range(4)]
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(g, want[i % 2]) for i, g in enumerate(got))


@pytest.mark.parametrize("M,ranks,launches", [
    (1, 1, 2), (14, 1, 2),        # few pairs, a cluster for each (and the sum)
    (1, 2, 2), (4, 2, 2),         # half of them here
    (14, 2, 3),                   # clusters narrow enough for all that may stay take longer than plan, layer and sum
    (2, 4, 2), (14, 4, 2), (30, 4, 3),
    (1, 8, 2), (6, 8, 3), (14, 8, 3),
])
def test_fused_moe_few_pairs_of_one_rank(M, ranks, launches):
    # which path an expert-parallel rank takes goes by the pairs that are expected to be its own, not by all of them
    import synth
    from dgx_vllm_b200 import _lib, sparse_fp4_v7 as sp7
    from dgx_vllm_b200.moe_ep import expert_map_for_rank
    from util import expert_fetch, gpu_quantize_fn, rel_err
    keys, E, H, I = ("comp_T", "meta_T", "scale_T", "g_scales"), 512, 2048, 512
    w13 = synth.make_sparse_experts(64, 2 * I, H, 1, "cuda", gpu_quantize_fn)
    w2 = synth.make_sparse_experts(64, H, I, 2, "cuda", gpu_quantize_fn)
    w13, w2 = ({k: w[k].repeat(E // ranks // 64, *[1] * (w[k].dim() - 1)) for k in keys} for w in (w13, w2))      # the same 64 again
    tw, ids = synth.make_routing(M, E, 10, 3 + M, "cuda")
    emap = expert_map_for_rank(E, ranks, ranks - 1, "cuda") if ranks > 1 else None
    hidden = synth.make_hidden(M, H, 4, "cuda")
    layer = sp7.FusedSparseMoE(*[w13[k] for k in keys], *[w2[k] for k in keys], I, expert_map=emap)
    n0 = _lib.lib().b200fp4_launch_count()
    out = layer(hidden, tw, ids)
    assert _lib.lib().b200fp4_launch_count() == n0 + launches and sp7.last_moe_status() == 0
    local = ids if emap is None else emap[ids.long()]
    ref = oracle.fused_sparse_moe_by_expert(hidden.float().cpu().numpy(), tw.cpu().numpy(), local.cpu().numpy(), expert_fetch(w13, w2), I)
    assert np.abs(to_np(out) - ref).max() <= 1e-2 * max(np.abs(ref).max(), 1e-6)


@pytest.mark.parametrize("M,topk,E,ranks,H,I,dtype", [
    (1, 4, 16, 1, 5760, 128, torch.bfloat16),      # the widest row that the layer takes: many threads bring in a second 16-byte piece of it
    (2, 3, 32, 2, 4224, 256, torch.float16),       # a few threads have a second one
    (3, 2, 64, 4, 256, 1024, torch.bfloat16),      # two pairs in four elsewhere, K short in gate_up and long in down
])
def test_fused_moe_few_pairs_in_records(M, topk, E, ranks, H, I, dtype):
    # rows, ids and weights apart by the length of a dispatch record; the same result as from tensors of their own
    import synth
    from dgx_vllm_b200 import _lib, sparse_fp4_v7 as sp7
    from dgx_vllm_b200._torch_util import workspace
    from dgx_vllm_b200.moe_ep import expert_map_for_rank
    from util import expert_fetch, gpu_quantize_fn, rel_err
    L, keys, here = _lib.lib(), ("comp_T", "meta_T", "scale_T", "g_scales"), E // ranks
    w13 = synth.make_sparse_experts(here, 2 * I, H, 1, "cuda", gpu_quantize_fn)
    w2 = synth.make_sparse_experts(here, H, I, 2, "cuda", gpu_quantize_fn)
    tw, ids = synth.make_routing(M, E, topk, 3, "cuda")
    ids[0, 0] = (ranks - 1) * here                  # at least one pair is this rank's
    hidden, emap = synth.make_hidden(M, H, 4, "cuda", dtype), expert_map_for_rank(E, ranks, ranks - 1, "cuda")
    code, R = (_lib.BF16 if dtype == torch.bfloat16 else _lib.F16), L.b200fp4_ep_record_bytes(H, topk)
    rec = torch.empty(M * R, dtype=torch.uint8, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(L.b200fp4_ep_pack(hidden.data_ptr(), ids.data_ptr(), tw.data_ptr(), M, H, topk, 1, rec.data_ptr(), st), "pack")
    out = torch.full((M, H), 7.0, dtype=dtype, device="cuda")
    ws = workspace(torch.device("cuda", torch.cuda.current_device()), L.b200fp4_fused_moe_workspace_bytes(M, topk, H, I, here))
    n0 = L.b200fp4_launch_count()
    _lib.check(L.b200fp4_fused_sparse_moe_records(
        rec.data_ptr(), R, code, emap.data_ptr(), E, *[w13[k].data_ptr() for k in keys], w13["scale_T"].shape[1],
        *[w2[k].data_ptr() for k in keys], w2["scale_T"].shape[1], out.data_ptr(), code, M, topk, H, I, here, _lib.SPARSE_META_ORDERED,
        ws.data_ptr(), ws.numel(), st), "records")
    assert L.b200fp4_launch_count() == n0 + 2
    want = sp7.fused_sparse_moe_v7(hidden, tw, ids, emap, *[w13[k] for k in keys], *[w2[k] for k in keys], I, False)
    assert L.b200fp4_launch_count() == n0 + 4 and sp7.last_moe_status() == 0
    assert torch.equal(out, want)
    ref = oracle.fused_sparse_moe_by_expert(hidden.float().cpu().numpy(), tw.cpu().numpy(), emap[ids.long()].cpu().numpy(),
                                            expert_fetch(w13, w2), I)
    assert rel_err(to_np(out), ref) < 1e-2


@pytest.mark.parametrize("M,N,K,launches,in_graph", [
    (44, 512, 512, 1, 1), (45, 512, 512, 1, 2), (60, 512, 512, 1, 2), (61, 512, 512, 2, 2), (64, 1024, 4096, 1, 1), (24, 4096, 2048, 1, 1),
    (25, 4096, 2048, 2, 2), (56, 2048, 1536, 1, 1), (57, 2048, 1536, 2, 2), (44, 3200, 1024, 1, 1), (45, 3200, 1024, 1, 2), (24, 9600, 1024, 1, 1),
    (28, 9600, 1024, 1, 2), (29, 9600, 1024, 2, 2), (32, 14336, 512, 1, 1), (33, 14336, 512, 1, 2), (48, 14336, 512, 1, 2), (49, 14336, 512, 2, 2),
    (16, 14336, 4096, 1, 1), (17, 14336, 4096, 2, 2),
])
def test_linear_path(M, N, K, launches, in_graph):
    # one kernel for few tokens, quantizer and GEMM where those are the faster ones: sooner in a graph, where a launch costs the host nothing
    from dgx_vllm_b200 import _lib, cutlass_scaled_fp4_mm, scaled_fp4_quant
    from dgx_vllm_b200.ops import last_gemm_status, nvfp4_linear
    x, gx, wc, ws, alpha = _linear_operands(M, N, K, M + N)
    n0 = _lib.lib().b200fp4_launch_count()
    out = nvfp4_linear(x, gx, wc, ws, alpha)
    assert _lib.lib().b200fp4_launch_count() == n0 + launches and last_gemm_status() == 0
    xc, xs = scaled_fp4_quant(x, gx)
    assert torch.equal(out, cutlass_scaled_fp4_mm(xc, wc, xs, ws, alpha, torch.bfloat16))
    graph, captured = torch.cuda.CUDAGraph(), torch.zeros_like(out)
    with torch.cuda.graph(graph):
        n0 = _lib.lib().b200fp4_launch_count()
        nvfp4_linear(x, gx, wc, ws, alpha, out=captured)
        assert _lib.lib().b200fp4_launch_count() == n0 + in_graph
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(captured, out)


@pytest.mark.parametrize("M,N,K", [
    (1, 128, 64), (4, 512, 512), (5, 512, 512),               # short K: the few-token kernel for up to four tokens, never in a graph
    (16, 520, 1088), (17, 520, 1088), (24, 512, 1536),        # few CTAs: up to 16 or 24
    (8, 4096, 4096), (9, 4096, 4096), (8, 4096, 2048),        # clusters that nearly fill the chip; the first in a graph too
    (8, 9600, 2112), (16, 14336, 4096),                       # K not split
])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gemm_of_few_tokens_eager_and_captured(M, N, K, dtype):
    # the two may be different kernels: both within one rounding to 16 bits and the f32 sum over K of the exact product of the codes
    from dgx_vllm_b200 import cutlass_scaled_fp4_mm, scaled_fp4_quant
    from dgx_vllm_b200.ops import last_gemm_status
    x, gx, wc, ws, alpha = _linear_operands(M, N, K, M + K)
    xc, xs = scaled_fp4_quant(x, gx)
    outs = [cutlass_scaled_fp4_mm(xc, wc, xs, ws, alpha, dtype, tile_n=t) for t in (0, 128)]
    assert last_gemm_status() == 0
    graph, out = torch.cuda.CUDAGraph(), torch.full((M, N), 7.0, dtype=dtype, device="cuda")
    with torch.cuda.graph(graph):
        cutlass_scaled_fp4_mm(xc, wc, xs, ws, alpha, dtype, out=out)
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()

    def deq(codes, sf, rows):
        lin = oracle.sf_swizzled_to_linear(to_np(sf.view(torch.uint8)).reshape(-1), rows, K // 16)
        return torch.from_numpy(oracle.dequantize(to_np(codes), lin, 1.0)).cuda().double()

    a, b = deq(xc, xs, M), deq(wc, ws, N)
    ref, size = (a @ b.t()) * alpha.double(), (a.abs() @ b.abs().t()) * alpha.double()
    bound = 2.0 ** (-8 if dtype == torch.bfloat16 else -11) * ref.abs() + 2.0 ** -20 * size + 2.0 ** -24
    for o in outs + [out]:
        assert bool(((o.double() - ref).abs() <= bound).all())
