"""Edges of the kernels' tiles, splits and dispatch rules on one GPU, against plain PyTorch."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import torch.distributed as dist

    import iris_b200 as iris

    torch.cuda.set_device(0)
    own = not dist.is_initialized()
    if own:
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1, device_id=torch.device("cuda", 0))
    c = iris.iris(1 << 30)
    yield c
    c.close()
    if own:
        dist.destroy_process_group()


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


# ------------------------------------------------------------------------------------ quantiser
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("M,K,pad", [(1, 16, 0), (3, 128, 0), (130, 1000, 0), (257, 384, 8), (64, 1152, 4), (5, 200, 1), (128, 2048, 0)])
def test_quantiser_matches_pytorch_bytes(dtype, M, K, pad):
    """Values, fp32 scales and packed atoms equal the PyTorch quantiser byte for byte (power-of-two scales: the
    divisions are exact), for ragged rows and columns and for row pitches of every alignment."""
    from iris_b200.ops.gemm_fp8 import pack_scales_a, quantize_1x128, quantize_activation

    x = (torch.randn(M, K + pad, device="cuda", generator=_gen(M + K)) * 3).to(dtype)[:, pad // 2: pad // 2 + K]
    got = quantize_activation(x)
    q, s = quantize_1x128(x, pow2=True)
    assert torch.equal(got.q.view(torch.uint8), q.view(torch.uint8))
    assert torch.equal(got.scale, s)
    assert torch.equal(got.sf(), pack_scales_a(s))


# ------------------------------------------------------------------------------------ activation passes
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("name", ["silu", "gelu"])
@pytest.mark.parametrize("shape", [(1, 1), (3, 5), (1, 8), (7, 2048), (129, 1000)])
def test_activation_passes_match_fp64(dtype, name, shape):
    """h and dpre against the fp64 expressions: one rounding of each result to the 16-bit type (unit roundoff 2^-8
    for bf16's 8 significant bits, 2^-11 for fp16's 11), plus fp32 rounding of terms that cancel near act' = 0."""
    from iris_b200.models.tp_mlp import _act_backward, _act_forward

    g = _gen(shape[0] * 7 + shape[1])
    pre = (torch.randn(*shape, device="cuda", generator=g) * 4).to(dtype)
    dh = torch.randn(*shape, device="cuda", generator=g).to(dtype)
    x = pre.double().requires_grad_(True)
    y = torch.nn.functional.silu(x) if name == "silu" else torch.nn.functional.gelu(x, approximate="tanh")
    (want_g,) = torch.autograd.grad(y, x, dh.double())
    dpre, h = _act_backward(name, dh, pre)
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    tiny = 2.0 ** -25 if dtype == torch.float16 else 0.0          # half the spacing of fp16 subnormals
    for got, want in ((h, y.detach()), (dpre, want_g), (_act_forward(name, pre), y.detach())):
        assert ((got.double() - want).abs() <= ulp * want.abs() + 4e-6 * (1 + dh.double().abs()) + tiny).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,KB", [(1, 8), (3, 7), (127, 16), (129, 13), (130, 9), (300, 24), (257, 40), (2050, 8)])
def test_quantiser_by_rows_equals_the_general_one(dtype, M, KB):
    """Aligned rows of whole blocks go eight blocks of a row to a warp (7, 8, 13, 16 ... blocks; 9 do not); the same values a few elements off the
    boundary take the general kernel: every value, scale and scale atom has to be the same, with NaN, infinities and zeros among them."""
    from iris_b200.ops import quantize_activation

    K = KB * 128
    base = torch.zeros(M * (K + 8) + 8, device="cuda", dtype=dtype)
    x = torch.randn(M, K, device="cuda", generator=_gen(M + KB)) * torch.logspace(-6, 4, M, device="cuda")[:, None]
    x[0, :128] = 0
    x[M // 2, 5], x[M - 1, K - 1], x[M // 3, K // 2] = float("nan"), float("inf"), -float("inf")
    x = x.to(dtype)
    off = base[4:4 + M * K].view(M, K)                # 8 or 16 bytes off a 16-byte boundary's multiple: rows take 8-byte loads at most
    if dtype == torch.float32:
        off = base[2:2 + M * K].view(M, K)
    off.copy_(x)
    assert x.data_ptr() % 16 == 0 and off.data_ptr() % 16 == 8
    a, b = quantize_activation(x), quantize_activation(off)
    assert torch.equal(a.q.view(torch.uint8), b.q.view(torch.uint8)) and torch.equal(a.scale, b.scale) and torch.equal(a.sf(), b.sf())


@pytest.mark.parametrize("M", [64, 65, 100, 128, 129])
@pytest.mark.parametrize("N,K", [(1000, 2048), (1544, 3000), (2048, 4096), (3072, 2112), (4096, 2048), (4744, 4096)])
@pytest.mark.parametrize("linear", [False, True])
def test_few_rows_on_both_ring_depths(M, N, K, linear):
    """Both sides of the rules that give a CTA an SM of its own (64 / 65 and 128 / 129 rows; up to 12 column tiles, 24 to 37, others), ragged
    tiles and K blocks. One rounding to bf16 (2^-8 of the value); fp32 sums of K products whose magnitudes add up to S, in any order: K 2^-24 S."""
    from iris_b200.ops import matmul

    g = _gen(M + N + K)
    a = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    b = w.t() if linear else w.t().contiguous()
    got, want = matmul(a, b).double(), a.double() @ w.double().t()
    sums = a.double().abs() @ w.double().abs().t()
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + K * 2.0 ** -24 * sums).all()


def _e4m3_operands(M, N, K, seed):
    """Values and power-of-two scales that differ from block to block: a scale atom or a tile taken for another shows."""
    from iris_b200.ops.gemm_fp8 import quantize_1x128, quantize_128x128

    g = _gen(seed)
    spread = lambda *sh: torch.exp2(torch.randint(-3, 4, sh, device="cuda", generator=g).float())  # noqa: E731
    kb = -(-K // 128)
    x = torch.randn(M, K, device="cuda", generator=g) * spread(M, kb).repeat_interleave(128, 1)[:, :K]
    w = torch.randn(N, K, device="cuda", generator=g) * spread(-(-N // 128), kb).repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)[:, :K]
    return quantize_1x128(x, pow2=True), quantize_128x128(w, pow2=True)


def _e4m3_pairs(M, N, K):
    """Whether the plan takes CTA pairs when nothing is asked for."""
    import ctypes as C

    from iris_b200 import _lib

    d = _lib.IrisGemmDesc()
    d.op, d.M, d.N, d.K, d.dtype, d.in_dtype, d.b_kmajor = _lib.GEMM_LOCAL, M, N, K, _lib.DTYPE_CODE[torch.bfloat16], _lib.DTYPE_CODE[torch.float8_e4m3fn], 1
    d.ctx.world = 1
    out = [C.c_uint64(), C.c_uint64(), C.c_uint64(), C.c_int32(), C.c_int32()]
    assert _lib.kernels().iris_gemm_workspace(C.byref(d), *[C.byref(o) for o in out]) == 0
    return bool(out[4].value)


@pytest.mark.parametrize("M", [1, 16, 129, 300, 385])
@pytest.mark.parametrize("N,K,by_rule", [(3656, 8192, True), (8200, 4224, True), (456, 4096, True), (1000, 1168, False), (224, 128, False)])
def test_e4m3_pairs_with_ragged_tiles(M, N, K, by_rule):
    """CTA pairs with rows for one of the two CTAs only, odd counts of 128-row tiles, ragged last columns and K blocks: where the rule chooses them,
    where they are asked for, and against single tiles. fp32 sums of K exact products in K order in both: the same values; against 64 bits one
    rounding to bf16 (2^-8 of it) and the sums' own, K 2^-24 of the magnitudes added up."""
    from iris_b200.ops.gemm_fp8 import dequantize, matmul_fp8_blockscaled, pack_scales_a, pack_scales_b

    (aq, asc), (bq, bsc) = _e4m3_operands(M, N, K, M + N)
    run = lambda two_sm: matmul_fp8_blockscaled(aq, pack_scales_a(asc), bq, pack_scales_b(bsc, N, 224), two_sm=two_sm)  # noqa: E731
    assert _e4m3_pairs(M, N, K) == (by_rule and not (M == 1 and N == 8200))
    pairs, single, chosen = run(True), run(False), run(None)
    a, b = dequantize(aq, asc, 1).double(), dequantize(bq, bsc, 128).double()
    want, sums = a @ b.t(), a.abs() @ b.abs().t()
    assert ((pairs.double() - want).abs() <= 2.0 ** -8 * want.abs() + K * 2.0 ** -24 * sums).all()
    assert torch.equal(pairs, single) and torch.equal(chosen, pairs)


# ------------------------------------------------------------------------------------ kernels that start behind their predecessor
@pytest.mark.parametrize("rows", [16, 300, 2000])
def test_chains_of_early_started_kernels(ctx, rows):
    """Every kernel that is launched before its predecessor has finished, in chains where each reads what the one in front wrote and
    buffers are written again at once, among ordinary kernels, with a second stream joined in, plain and as a CUDA graph: the bits
    of the same calls with the device idle in between."""
    from iris_b200.models import FlashDecodeLayer, RingAttention
    from iris_b200.ops import matmul, quantize_activation, quantize_weight

    g = _gen(rows)
    r = lambda *sh: torch.randn(*sh, device="cuda", generator=g) * sh[-1] ** -0.5  # noqa: E731
    D = 1024
    w1, w2, wq = r(D, D).bfloat16().t(), r(D, D).bfloat16(), quantize_weight(r(D, D))
    cache = [torch.randn(64, 16, 2, 128, device="cuda", generator=g).bfloat16() for _ in range(2)]
    table, lens = torch.randperm(64, device="cuda", generator=g).int().view(2, 32), torch.tensor([[511, 77]], device="cuda", dtype=torch.int32)
    mark = ctx.heap_mark()
    dec, att = FlashDecodeLayer(ctx, 8, 2, 128, max_batch=2), RingAttention(ctx, rows, 8, 2)
    x0 = torch.randn(rows, D, device="cuda", generator=g).bfloat16()
    x, h, y = x0.clone(), torch.empty_like(x0), torch.empty_like(x0)
    side = torch.cuda.Stream()

    def chain(sync):
        gap = torch.cuda.synchronize if sync else (lambda: None)
        x.copy_(x0)
        for _ in range(3):
            gap(); matmul(x, w1, out=h)
            gap(); matmul(h, w2, out=x)
            gap(); a = quantize_activation(x)
            gap(); matmul(a, wq, out=y)
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                gap(); matmul(y, w2, out=h)
            torch.cuda.current_stream().wait_stream(side)
            gap(); o = att(h.view(rows, 8, 128), x.view(rows, 8, 128)[:, :2].contiguous(), y.view(rows, 8, 128)[:, 2:4].contiguous(), causal=True)
            gap(); d = dec(o[:2], *cache, lens, table)
            gap(); x[:2] = d.view(2, D)
            gap(); x.mul_(4.0)
        return x.clone(), y.clone()

    want = chain(True)
    assert all(torch.isfinite(t.float()).all() and t.float().abs().max() > 0 for t in want)
    for _ in range(5):
        assert all(torch.equal(a, b) for a, b in zip(chain(False), want))
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        got = chain(False)
    for _ in range(3):
        graph.replay()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    del graph, got
    ctx.heap_release(mark)


# ------------------------------------------------------------------------------------ MoE on one rank
def _moe_weights(E, D, F, seed):
    g = _gen(seed)
    r = lambda *sh: (torch.randn(*sh, device="cuda", generator=g) * sh[1] ** -0.5).to(torch.bfloat16)  # noqa: E731
    return r(E, D, F), r(E, D, F), r(E, F, D)


@pytest.mark.parametrize("T,E,K", [(1, 8, 2), (37, 32, 8), (130, 64, 6), (5, 33, 4), (700, 130, 3), (64, 300, 16)])
def test_moe_one_rank_router_sort_gather(ctx, T, E, K):
    """Every template of the router (experts per lane 1 to 32), token counts around the block sizes, and experts
    masked with -inf or the type's lowest value. bf16 rounding of x, weights (exact here), hidden and the k
    outputs: each at most a relative 2^-8, in sum below 2e-2 of the output's 2-norm."""
    from iris_b200.models import MoELayer, reference_moe

    D, F = 256, 128
    wg, wu, wd = _moe_weights(E, D, F, E)
    mark = ctx.heap_mark()
    layer = MoELayer(ctx, D, F, E, K, max_tokens=T + 3, w_gate=wg, w_up=wu, w_down=wd)
    g = _gen(T)
    x = torch.randn(T, D, device="cuda", generator=g).to(torch.bfloat16)
    logits = torch.randn(T, E, device="cuda", generator=g)
    for masked in (None, float("-inf"), torch.finfo(torch.float32).min):
        if masked is not None:
            logits[:, : E // 2] = masked           # fewer than K experts stay in some of the cases
        y = layer(x, logits)
        want = reference_moe(x, logits, wg, wu, wd, K)
        assert ((y.float() - want).norm() / want.norm()).item() < 2e-2
        idx = layer.topk_idx[:T].long()
        assert (idx >= 0).all() and (idx < E).all() and all(len(set(r)) == K for r in idx.tolist())
    ctx.heap_release(mark)


@pytest.mark.parametrize("T", [256, 257])
def test_moe_e4m3_one_rank_preparation(ctx, T):
    """Both sides of the one-block preparation's limit, the kernels each is counted for, and no buffers for tokens that nobody
    sends. x, weights and hidden activations in e4m3 (4 significant bits, 2^-4 / sqrt(3) each): in sum below 0.1 of the
    output's 2-norm."""
    from iris_b200 import _lib
    from iris_b200.models import MoELayer, reference_moe

    E, D, F, K = 8, 256, 128, 2
    wg, wu, wd = _moe_weights(E, D, F, T)
    mark = ctx.heap_mark()
    layer = MoELayer(ctx, D, F, E, K, max_tokens=T, w_gate=wg, w_up=wu, w_down=wd, fp8=True)
    x = torch.randn(T, D, device="cuda", generator=_gen(T)).to(torch.bfloat16)
    logits = torch.randn(T, E, device="cuda", generator=_gen(T + 1))
    before = _lib.LAUNCHES.get("MoE forward launch", 0)
    y = layer(x, logits)
    assert _lib.LAUNCHES["MoE forward launch"] - before == (5 if T <= _lib.kernels().iris_moe_prep_max_tokens() else 8) == (5 if T == 256 else 8)
    want = reference_moe(x, logits, wg, wu, wd, K)
    assert ((y.float() - want).norm() / want.norm()).item() < 0.1 and layer.xq is None and layer.x_sf is None
    ctx.heap_release(mark)


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("T,E,K,D,F", [(1, 4, 2, 256, 128), (16, 2, 2, 512, 256), (17, 3, 1, 256, 384), (64, 2, 2, 256, 128), (65, 2, 2, 256, 128),
                                       (240, 2, 2, 512, 128), (241, 2, 2, 256, 256), (256, 3, 3, 256, 128), (257, 2, 2, 512, 128), (513, 5, 2, 256, 128),
                                       (1000, 40, 1, 256, 128), (1500, 8, 4, 1024, 512)])
def test_moe_one_rank_token_tiles(ctx, fp8, T, E, K, D, F):
    """Token tiles of every padded size: experts that take every token (E = K: T rows each, both sides of the tile limits 64, 240 and
    256), experts without tokens, a layer made for more tokens than the call has. Rows of the buffers behind an expert's last
    tile hold other experts' rows. Bounds as in the two tests above; the e4m3 layer is compared over its dequantised weights."""
    from iris_b200.models import MoELayer, reference_moe
    from iris_b200.ops.gemm_fp8 import dequantize, quantize_128x128

    wg, wu, wd = _moe_weights(E, D, F, T + E)
    mark = ctx.heap_mark()
    layer = MoELayer(ctx, D, F, E, K, max_tokens=T + 300, w_gate=wg, w_up=wu, w_down=wd, fp8=fp8)
    if fp8:
        deq = lambda w: torch.stack([dequantize(*quantize_128x128(m.t().contiguous().float(), pow2=True), 128).t() for m in w])  # noqa: E731
        wg, wu, wd = deq(wg), deq(wu), deq(wd)
    x = torch.randn(T, D, device="cuda", generator=_gen(T)).to(torch.bfloat16)
    logits = torch.randn(T, E, device="cuda", generator=_gen(T + 1))
    if K < E:
        logits[:, E // 2:] -= 1.5 * torch.arange(E - E // 2, device="cuda")        # crowded and empty experts
    y = layer(x, logits)
    want = reference_moe(x, logits, wg, wu, wd, K)
    assert ((y.float() - want).norm() / want.norm()).item() < (0.1 if fp8 else 2e-2)
    worst = ((y.float() - want).norm(dim=1) / want.norm(dim=1)).max().item()         # no row is another's
    assert worst < (0.2 if fp8 else 4e-2), worst
    assert torch.equal(y, layer(x, logits))
    ctx.check()
    ctx.heap_release(mark)


@pytest.mark.parametrize("T,fp8", [(20, True), (20, False), (300, True)])
def test_moe_one_rank_in_a_cuda_graph(ctx, T, fp8):
    """The launches that start behind their predecessors, captured: a replay on new inputs gives the bits of a plain call."""
    from iris_b200.models import MoELayer

    E, D, F, K = 8, 512, 256, 2
    mark = ctx.heap_mark()
    layer = MoELayer(ctx, D, F, E, K, max_tokens=T, **dict(zip(("w_gate", "w_up", "w_down"), _moe_weights(E, D, F, 3))), fp8=fp8)
    x, logits, out = torch.zeros(T, D, device="cuda", dtype=torch.bfloat16), torch.zeros(T, E, device="cuda"), torch.zeros(T, D, device="cuda", dtype=torch.bfloat16)
    layer(x, logits, out=out)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(3):                       # the next call's first kernel follows the last call's reduction
            layer(x, logits, out=out)
    for seed in (1, 2):
        x.copy_(torch.randn(T, D, device="cuda", generator=_gen(seed)))
        logits.copy_(torch.randn(T, E, device="cuda", generator=_gen(seed + 10)))
        graph.replay()
        got = out.clone()
        assert got.abs().max() > 0 and torch.equal(got, layer(x, logits))
    del graph
    ctx.heap_release(mark)


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("T", [3, 70])
def test_moe_one_rank_swiglu_divides_exactly(ctx, fp8, T):
    """Gates around -88, where 1 + exp(-gate) lies above 2^126 and a fast division returns zero, against up values of 2^120. Products and sums are exact
    here; __expf is within 105 ulp (1.3e-5) there; bf16 rounds the hidden value and the output (2^-9 each), e4m3 the hidden value (2^-4)."""
    from iris_b200.models import MoELayer

    D, F = 256, 128
    gate = torch.full((F,), -88.0, device="cuda") if fp8 else -80.0 - 0.5 * (torch.arange(F, device="cuda") % 18)
    w_gate, w_up, w_down = torch.zeros(1, D, F, device="cuda"), torch.zeros(1, D, F, device="cuda"), torch.zeros(1, F, D, device="cuda")
    w_gate[0, 0], w_up[0, 0] = gate, 2.0 ** 120
    w_down[0, :, :F] = torch.eye(F, device="cuda")
    x = torch.zeros(T, D, device="cuda", dtype=torch.bfloat16)
    x[:, 0] = 1
    mark = ctx.heap_mark()
    layer = MoELayer(ctx, D, F, 1, 1, max_tokens=T, w_gate=w_gate.bfloat16(), w_up=w_up.bfloat16(), w_down=w_down.bfloat16(), fp8=fp8)
    got = layer(x, torch.zeros(T, 1, device="cuda"))[:, :F].double()
    g = gate.double()
    want = g / (1 + torch.exp(-g)) * 2.0 ** 120
    assert ((got - want).abs() <= ((2.0 ** -4 if fp8 else 0.0) + 2.0 ** -8 + 2e-5) * want.abs()).all()
    ctx.heap_release(mark)


@pytest.mark.parametrize("T,fp8", [(48, True), (48, False), (700, True), (700, False)])
def test_moe_one_rank_many_units_per_pair(ctx, T, fp8):
    """Four or more units per CTA pair in both grouped GEMMs, and K blocks (22 and 11 in e4m3, 44 and 22 in bf16) that pass every ring (9, 10, 5 and 6 stages)
    more than once without being a multiple: accumulator buffers, barrier phases and the exchanged magnitudes are used again and again. Other inputs
    in between. Bounds as in test_moe_one_rank_token_tiles."""
    from iris_b200.models import MoELayer, reference_moe
    from iris_b200.ops.gemm_fp8 import dequantize, quantize_128x128

    E, K, D, F = 32, 8, 2816, 1408
    wg, wu, wd = _moe_weights(E, D, F, T)
    mark = ctx.heap_mark()
    layer = MoELayer(ctx, D, F, E, K, max_tokens=T, w_gate=wg, w_up=wu, w_down=wd, fp8=fp8)
    if fp8:
        deq = lambda w: torch.stack([dequantize(*quantize_128x128(m.t().contiguous().float(), pow2=True), 128).t() for m in w])  # noqa: E731
        wg, wu, wd = deq(wg), deq(wu), deq(wd)
    calls = [(torch.randn(T, D, device="cuda", generator=_gen(i)).to(torch.bfloat16), torch.randn(T, E, device="cuda", generator=_gen(i + 50))) for i in range(3)]
    first = []
    for x, logits in calls:
        y, want = layer(x, logits), reference_moe(x, logits, wg, wu, wd, K)
        # 32 x 11 weight tiles of 256 rows each (down: the same number), times the token tiles of the experts in use, on 74 pairs
        assert layer.tile_prefix[E].item() * 11 >= 4 * 74
        assert ((y.float() - want).norm() / want.norm()).item() < (0.1 if fp8 else 2e-2)
        assert ((y.float() - want).norm(dim=1) / want.norm(dim=1)).max().item() < (0.2 if fp8 else 4e-2)
        first.append(y)
    for _ in range(3):
        outs = [layer(x, logits) for x, logits in calls]
        assert all(torch.equal(a, b) for a, b in zip(outs, first))
    ctx.check()
    ctx.heap_release(mark)


@pytest.mark.parametrize("T", [40, 300])
def test_moe_one_rank_weights_that_are_not_k_major(ctx, T):
    """What only a C caller asks for (weights_kmajor 0: w13 [El, D, 2F], w2 [El, F, D]): the grouped GEMM of several ranks, on one. Sums in the same order as with
    K-major weights up to the tile's shape, so both are within the bf16 bounds above of the reference."""
    import ctypes as C

    from iris_b200 import _lib
    from iris_b200.models import MoELayer, reference_moe
    from iris_b200.models.moe import fuse_gate_up

    E, K, D, F = 6, 2, 512, 256
    wg, wu, wd = _moe_weights(E, D, F, T)
    mark = ctx.heap_mark()
    layer = MoELayer(ctx, D, F, E, K, max_tokens=T, w_gate=wg, w_up=wu, w_down=wd)
    x, logits = torch.randn(T, D, device="cuda", generator=_gen(T)).to(torch.bfloat16), torch.randn(T, E, device="cuda", generator=_gen(1))
    out, w13, w2 = torch.empty_like(x), fuse_gate_up(wg, wu), wd.contiguous()
    d = layer._descriptor(x, logits, out)
    d.weights_kmajor, d.w13, d.w2 = 0, w13.data_ptr(), w2.data_ptr()
    for _ in range(2):
        assert layer._lib().iris_moe_forward(C.byref(d), C.c_void_p(_lib.current_stream_ptr())) == 0
        want = reference_moe(x, logits, wg, wu, wd, K)
        assert ((out.float() - want).norm() / want.norm()).item() < 2e-2
        assert ((out.float() - want).norm(dim=1) / want.norm(dim=1)).max().item() < 4e-2
        y = layer(x, logits)                       # and the layer's own form between the two
        assert ((y.float() - want).norm() / want.norm()).item() < 2e-2
        out.zero_()
    ctx.check()
    ctx.heap_release(mark)


@pytest.mark.parametrize("T,fp8", [(24, True), (24, False), (300, True), (300, False)])
def test_moe_among_other_early_started_kernels(ctx, T, fp8):
    """The MoE layer between GEMMs, the quantiser, decode and elementwise kernels, each reading what the one in front wrote, plain and as a CUDA graph: the bits of
    the same calls with the device idle in between."""
    from iris_b200.models import FlashDecodeLayer, MoELayer
    from iris_b200.ops import matmul, quantize_activation, quantize_weight

    g, D, E = _gen(T), 1024, 8
    r = lambda *sh: torch.randn(*sh, device="cuda", generator=g) * sh[-1] ** -0.5  # noqa: E731
    w1, w2, wr, wq = r(D, D).bfloat16().t(), r(D, D).bfloat16(), r(E, D).bfloat16().t(), quantize_weight(r(D, D))
    cache = [torch.randn(64, 16, 2, 128, device="cuda", generator=g).bfloat16() for _ in range(2)]
    table, lens = torch.randperm(64, device="cuda", generator=g).int().view(2, 32), torch.tensor([[511, 77]], device="cuda", dtype=torch.int32)
    mark = ctx.heap_mark()
    dec = FlashDecodeLayer(ctx, 8, 2, 128, max_batch=2)
    moe = MoELayer(ctx, D, 512, E, 2, max_tokens=T, **dict(zip(("w_gate", "w_up", "w_down"), _moe_weights(E, D, 512, 5))), fp8=fp8)
    x0 = torch.randn(T, D, device="cuda", generator=g).bfloat16()
    x, h, y, logits = x0.clone(), torch.empty_like(x0), torch.empty_like(x0), torch.empty(T, E, device="cuda", dtype=torch.bfloat16)

    def chain(sync):
        gap = torch.cuda.synchronize if sync else (lambda: None)
        x.copy_(x0)
        for _ in range(3):
            gap(); matmul(x, w1, out=h)
            gap(); matmul(h, wr, out=logits)
            gap(); moe(h, logits, out=y)                       # tokens straight from a GEMM
            gap(); matmul(y, w2, out=x)                        # and its sum straight into one
            gap(); a = quantize_activation(x)
            gap(); matmul(a, wq, out=h)
            gap(); moe(h, logits, out=y)
            gap(); moe(y, logits, out=x)                       # back to back, tokens from the reduction in front
            gap(); d = dec(x[:2].view(2, 8, 128), *cache, lens, table)
            gap(); x[:2] = d.view(2, D)
            gap(); x.mul_(8.0)
        return x.clone(), y.clone()

    want = chain(True)
    assert all(torch.isfinite(t.float()).all() and t.float().abs().max() > 0 for t in want)
    for _ in range(5):
        assert all(torch.equal(a, b) for a, b in zip(chain(False), want))
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        got = chain(False)
    for _ in range(3):
        graph.replay()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    del graph, got
    ctx.heap_release(mark)


# ------------------------------------------------------------------------------------ attention on one rank
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("S,Hq,Hkv", [(1, 2, 2), (64, 4, 2), (127, 8, 2), (128, 3, 1), (129, 4, 4), (257, 6, 2), (384, 5, 5), (1000, 8, 8), (2500, 16, 2),
                                      (300, 2, 1), (640, 8, 2), (2304, 4, 2), (4700, 4, 4),
                                      (2500, 8, 8), (2300, 9, 3), (2400, 9, 3), (2300, 18, 3), (4200, 9, 3), (4300, 9, 3)])
@pytest.mark.parametrize("causal", [False, True])
def test_attention_any_length_and_group(ctx, dtype, S, Hq, Hkv, causal):
    """Every form of the dispatch, lengths on both sides of the 128-row tiles, against fp32 attention: the mma.sync CTAs (up to
    128 tokens); one query tile whose keys two softmax groups share (at most as many query tiles as SMs, 148, under a causal
    mask twice as many: up to (4700, 4, 4); odd and even numbers of key tiles, one in the first causal tile); two heads of an
    even group per item ((2500, 16, 2), (2300, 18, 3)); two neighbouring query tiles of one head ((2500, 8, 8), (2300, 9, 3) with
    full attention, (4300, 9, 3) with either), the last item of an odd count with one tile ((2400, 9, 3), (4200, 9, 3)). P and the
    output are rounded to 16 bits: |error| <= 2 u max|v| with u = 2^-8 (bf16) or 2^-11 (fp16), and max|v| < 6 here.
    The scores are scaled up so that rows move their maximum late (the rescaling of O) as well as early."""
    from iris_b200.models import RingAttention, reference_attention

    g = _gen(S + Hq)
    mk = lambda h, scale=1.0: (torch.randn(S, h, 128, device="cuda", generator=g) * scale).to(dtype)  # noqa: E731
    q, k, v = mk(Hq, 3.0), mk(Hkv), mk(Hkv).clamp(-6, 6)
    k = (k.float() * torch.linspace(0.1, 2.0, S, device="cuda")[:, None, None]).to(dtype)      # later keys score higher
    mark = ctx.heap_mark()
    layer = RingAttention(ctx, S, Hq, Hkv, dtype=dtype)
    out, lse = layer(q, k, v, causal=causal, return_lse=True)
    out2 = layer(q, k, v, causal=causal)                       # the other call parity
    want = reference_attention(q, k, v, causal)
    u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert (out.float() - want).abs().max().item() <= 2 * u * 6
    assert torch.equal(out, out2)
    kf = k.float().repeat_interleave(Hq // Hkv, dim=1)
    s = torch.einsum("qhd,khd->qhk", q.float(), kf) * 128 ** -0.5
    if causal:
        s = s.masked_fill((torch.arange(S, device="cuda")[None, :] > torch.arange(S, device="cuda")[:, None])[:, None, :], float("-inf"))
    assert (lse - torch.logsumexp(s, -1)).abs().max().item() < 1e-3
    ctx.heap_release(mark)


# ------------------------------------------------------------------------------------ decode
@pytest.mark.parametrize("tma", [None, False])
@pytest.mark.parametrize("B,Hq,Hkv,page,lens", [
    (1, 8, 1, 16, (1,)), (1, 8, 8, 64, (4096,)), (3, 8, 2, 16, (0, 63, 65)), (5, 32, 2, 32, (1, 256, 257, 5000, 0)),
    (2, 40, 1, 8, (4097, 129)), (33, 4, 4, 128, tuple(range(0, 33 * 37, 37))), (2, 64, 8, 24, (700, 2500)),
    (1100, 2, 1, 16, tuple((i * 7) % 90 for i in range(1100)))])
def test_decode_runs_cut_sequences_anywhere(ctx, tma, B, Hq, Hkv, page, lens):
    """Empty sequences, one tile, lengths around tile and run boundaries, many sequences per CTA and many CTAs per
    sequence, more sequences than one launch takes, head groups above 16 and page sizes without a TMA box. Probabilities and
    output are rounded to bf16 (2^-8 each) and |v| < 6: within 2 * 2^-8 * 6 of the fp32 result."""
    from iris_b200.models import FlashDecodeLayer, reference_decode

    g = _gen(B + Hq + page)
    L = max(max(lens), 1)
    blocks = -(-L // page)
    r = lambda *sh: torch.randn(*sh, device="cuda", generator=g).clamp(-6, 6).to(torch.bfloat16)  # noqa: E731
    q, k, v = r(B, Hq, 128), r(B * blocks, page, Hkv, 128), r(B * blocks, page, Hkv, 128)
    table = torch.randperm(B * blocks, device="cuda", generator=g).to(torch.int32).view(B, blocks)
    kv = torch.tensor([lens], dtype=torch.int32, device="cuda")
    mark = ctx.heap_mark()
    layer = FlashDecodeLayer(ctx, Hq, Hkv, max_batch=B, use_tma=tma)
    want, want_lse = reference_decode(q, k, v, kv[0], table)
    for splits in (64, 2, 1):
        layer.max_splits = splits
        out, lse = layer(q, k, v, kv, table, return_lse=True)
        assert (out.float() - want).abs().max().item() <= 2 * 2.0 ** -8 * 6
        seen = kv[0] > 0
        assert (lse[seen] - want_lse[seen]).abs().max().item() < 1e-3 if bool(seen.any()) else True
        assert torch.isneginf(lse[~seen]).all() and (out[~seen] == 0).all()
    ctx.heap_release(mark)


@pytest.mark.parametrize("B,Hq,Hkv,L,places", [(1, 8, 1, 32768, 41), (2, 16, 1, 20000, 41), (3, 128, 1, 4096, 9), (5, 64, 1, 9000, 9)])
def test_decode_fold_with_many_places(ctx, B, Hq, Hkv, L, places):
    """More places than a pass of the fold takes: above 40 where four threads share a column (few heads), above 8 where one does (more heads than two per SM).
    Bound as in the test above."""
    from iris_b200.models import FlashDecodeLayer, reference_decode

    g, page = _gen(B + L), 16
    blocks = -(-L // page)
    r = lambda *sh: torch.randn(*sh, device="cuda", generator=g).clamp(-6, 6).to(torch.bfloat16)  # noqa: E731
    q, k, v = r(B, Hq, 128), r(B * blocks, page, Hkv, 128), r(B * blocks, page, Hkv, 128)
    table = torch.randperm(B * blocks, device="cuda", generator=g).to(torch.int32).view(B, blocks)
    kv = torch.full((1, B), L, dtype=torch.int32, device="cuda")
    mark = ctx.heap_mark()
    layer = FlashDecodeLayer(ctx, Hq, Hkv, max_batch=B)
    out, lse = layer(q, k, v, kv, table, return_lse=True)
    splits = layer.num_splits(B, blocks * page)
    filled = ~torch.isneginf(layer.partial.view(-1)[:B * Hq * splits * 129].view(B * Hq, splits, 129)[:, :, 128])
    assert filled.sum(dim=1).max().item() >= places and (B * Hq > 2 * ctx.get_cu_count()) == (places == 9)
    want, want_lse = reference_decode(q, k, v, kv[0], table)
    assert (out.float() - want).abs().max().item() <= 2 * 2.0 ** -8 * 6 and (lse - want_lse).abs().max().item() < 1e-3
    ctx.heap_release(mark)


@pytest.mark.parametrize("B,L,low", [(1, 32768, 4096), (40, 2048, 1024)])
@pytest.mark.parametrize("at", [5, 200])
def test_decode_fold_ignores_places_of_no_weight(ctx, B, L, low, at):
    """The first `low` positions score 524 powers of two below the others and one of them has an infinite value: the runs they lie in (at most 640 of the
    4096 positions, 320 of the 1024) have weight zero and do not touch the result, in both forms of the fold. The others' values are equal: the
    output is that value, rounded (P and the output to 2^-8 each)."""
    from iris_b200.models import FlashDecodeLayer

    Hq, page = 8, 64
    blocks = L // page
    q = torch.zeros(B, Hq, 128, device="cuda", dtype=torch.bfloat16)
    k, v = torch.zeros(B, L, 128, device="cuda", dtype=torch.bfloat16), torch.zeros(B, L, 128, device="cuda", dtype=torch.bfloat16)
    q[..., 0], k[:, :low, 0] = 64, -64
    want = (1 + torch.arange(128, device="cuda") / 128).to(torch.bfloat16)
    v[:, low:] = want
    v[:, at] = float("inf")
    table = torch.arange(B * blocks, device="cuda", dtype=torch.int32).view(B, blocks)
    mark = ctx.heap_mark()
    layer = FlashDecodeLayer(ctx, Hq, 1, max_batch=B)
    out, lse = layer(q, k.view(B * blocks, page, 1, 128), v.view(B * blocks, page, 1, 128), torch.full((1, B), L, device="cuda", dtype=torch.int32), table,
                     return_lse=True)
    assert ((out.float() - want.float()).abs() <= 2 * 2.0 ** -8 * want.float()).all()
    assert (lse - torch.tensor(float(L - low)).log().item()).abs().max().item() < 1e-3
    ctx.heap_release(mark)


@pytest.mark.parametrize("tma", [None, False])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("soft_cap", [0.0, 30.0])
@pytest.mark.parametrize("Hq,Hkv", [(2, 2), (16, 2), (18, 2), (32, 2)])
def test_decode_is_exact_to_the_outputs_rounding(ctx, tma, dtype, soft_cap, Hq, Hkv):
    """Every instantiation (fill, type, groups up to 8 heads and above) against 64 bits. P is held as a rounded value and its
    remainder, so the output's rounding (u = 2^-8 or 2^-11 of it) is the error, plus 2^-14 of sum p |v| for the remainder's own
    rounding (2^-16) and fp32 scores and sums: a tile or page that were taken for another would show."""
    from iris_b200.models import FlashDecodeLayer

    g = _gen(Hq)
    lens, page = (700, 2500, 5000, 65), 16
    B, L = len(lens), max(lens)
    blocks = -(-L // page)
    r = lambda *sh: torch.randn(*sh, device="cuda", generator=g).to(dtype)  # noqa: E731
    q, k, v = r(B, Hq, 128), r(B * blocks, page, Hkv, 128), r(B * blocks, page, Hkv, 128)
    table = torch.randperm(B * blocks, device="cuda", generator=g).to(torch.int32).view(B, blocks)
    mark = ctx.heap_mark()
    layer = FlashDecodeLayer(ctx, Hq, Hkv, max_batch=B, soft_cap=soft_cap, dtype=dtype, use_tma=tma)
    out = layer(q, k, v, torch.tensor([lens], dtype=torch.int32, device="cuda"), table).double()
    u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for b, n in enumerate(lens):
        kb, vb = (t[table[b].long()].reshape(-1, Hkv, 128)[:n].repeat_interleave(Hq // Hkv, dim=1).double() for t in (k, v))
        s = torch.einsum("hd,khd->hk", q[b].double(), kb) * 128 ** -0.5
        p = torch.softmax(soft_cap * torch.tanh(s / soft_cap) if soft_cap else s, -1)
        want, size = torch.einsum("hk,khd->hd", p, vb), torch.einsum("hk,khd->hd", p, vb.abs())
        assert ((out[b] - want).abs() <= 1.01 * u * want.abs() + 2.0 ** -14 * size).all()
    ctx.heap_release(mark)


# ------------------------------------------------------------------------------------ few rows
@pytest.mark.parametrize("kmajor", [True, False])
@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (1, 1024, 64), (16, 136, 520), (17, 1032, 2048), (32, 3584, 72), (33, 264, 4096), (64, 2000, 3000),
                                   (65, 1024, 2048), (128, 640, 2056), (129, 256, 2816), (256, 4096, 2816), (200, 1544, 8192), (256, 128, 16384)])
def test_few_rows_gemm(kmajor, M, N, K):
    """Both sides of every step of the dispatch, ragged N and K, clusters of 1 to 8, biases of either kind and type, an
    output whose rows take no 8-byte stores. fp32 sums of bf16 products: |error| <= 2^-8 |C| (the output's rounding)
    plus a few 2^-24 sum |a||b|."""
    from iris_b200.ops import matmul

    for dtype, u in ((torch.bfloat16, 2.0 ** -8), (torch.float16, 2.0 ** -11)):
        g = _gen(M + N + K)
        A = torch.randn(M, K, device="cuda", generator=g).to(dtype)
        W = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).to(dtype)
        B = W.t() if kmajor else W.t().contiguous()
        ref = A.double() @ B.double()
        slack = 32 * 2.0 ** -24 * (A.double().abs() @ B.double().abs())
        wide = torch.empty(M, N + 3, device="cuda", dtype=dtype)
        for bias, dim in ((None, 1), (torch.randn(N, device="cuda", generator=g).to(dtype), 1), (torch.randn(N, device="cuda", generator=g), 1),
                          (torch.randn(M, device="cuda", generator=g).to(dtype), 0), (torch.randn(M + 1, device="cuda", generator=g)[1:], 0)):
            want = ref if bias is None else ref + (bias.double()[:, None] if dim == 0 else bias.double()[None, :])
            for out in (None, wide[:, 1:1 + N] if M <= 32 else None):
                C = matmul(A, B, bias=bias, bias_dim=dim, out=out)
                assert ((C.double() - want).abs() <= 1.01 * u * want.abs() + slack + 1e-7).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("offset", [0, 1, 4])
def test_column_bias_of_the_main_loop(dtype, offset):
    """The epilogue reads a column bias by 16-byte loads where it is aligned and one by one elsewhere, in fp32 and in
    the operands' type; N ends inside a 32-column chunk. Same bound as the test above."""
    from iris_b200.ops import matmul

    M, N, K = 300, 1000, 256
    g = _gen(offset)
    A = torch.randn(M, K, device="cuda", generator=g).to(dtype)
    B = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).to(dtype).t()
    u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    slack = 32 * 2.0 ** -24 * (A.double().abs() @ B.double().abs())
    for bdt in (dtype, torch.float32):
        bias = torch.randn(N + 8, device="cuda", generator=g).to(bdt)[offset:offset + N]
        want = A.double() @ B.double() + bias.double()[None, :]
        for kw in ({}, {"bn": 128}, {"bn": 224, "two_sm": False}, {"bn": 256, "two_sm": True}):
            assert ((matmul(A, B, bias=bias, **kw).double() - want).abs() <= 1.01 * u * want.abs() + slack + 1e-7).all()


@pytest.mark.parametrize("T,D,F", [(48, 1024, 512), (1, 256, 128), (130, 512, 384), (1000, 256, 512)])
def test_one_rank_ops_take_any_row_count(ctx, T, D, F):
    """Rows that are not a multiple of 128 on one rank: the op writes the output directly where it can, and still takes
    outputs it cannot write (another dtype, overlapping an input, unaligned rows)."""
    g = _gen(T)
    x = torch.randn(T, D, device="cuda", generator=g).to(torch.bfloat16)
    w1 = (torch.randn(F, D, device="cuda", generator=g) * D ** -0.5).to(torch.bfloat16).t()
    w2 = (torch.randn(D, F, device="cuda", generator=g) * F ** -0.5).to(torch.bfloat16).t()
    bias = torch.randn(T, device="cuda", generator=g).to(torch.bfloat16)
    h_ref = x.double() @ w1.double() + bias.double()[:, None]
    outs = [torch.empty(T, F, dtype=torch.bfloat16, device="cuda"), torch.empty(T, F + 1, dtype=torch.bfloat16, device="cuda")[:, 1:],
            torch.empty(T, F, dtype=torch.float32, device="cuda"), torch.empty(F, T, dtype=torch.bfloat16, device="cuda").t()]
    for h in outs:
        ctx.ops.all_gather_matmul(h, x, w1, bias=bias, shard_dim=0, async_op=True)
        assert ((h.double() - h_ref).norm() / h_ref.norm()).item() < 4e-3
    h = outs[0]
    y_ref = h.double() @ w2.double()
    for y in (torch.empty(T, D, dtype=torch.bfloat16, device="cuda"), torch.empty(T, D, dtype=torch.float32, device="cuda")):
        ctx.ops.matmul_reduce_scatter(y, h, w2, scatter_rows=True, async_op=True)
        assert ((y.double() - y_ref).norm() / y_ref.norm()).item() < 4e-3
    sq = (torch.randn(D, D, device="cuda", generator=g) * D ** -0.5).to(torch.bfloat16)
    want = x.double() @ sq.double()
    ctx.ops.all_gather_matmul(x, x, sq, shard_dim=0, async_op=True)          # in place
    assert ((x.double() - want).norm() / want.norm()).item() < 4e-3


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("op,kw", [("all_gather_matmul", {"shard_dim": 0}), ("all_gather_matmul", {"shard_dim": 1}), ("matmul_all_gather", {}),
                                   ("matmul_all_gather", {"scatter_cols": True}), ("matmul_all_reduce", {}), ("matmul_reduce_scatter", {"scatter_rows": True}),
                                   ("matmul_reduce_scatter", {})])
def test_fused_kernels_on_one_rank(ctx, op, kw, fp8):
    """With ``one_rank_fused`` an op's own kernel runs on one rank (its policy, epilogue, flags and double-buffered workspace), else
    a local GEMM, whose workspace reserves nothing on the heap but the sync block; both round one fp32 sum."""
    from iris_b200.ops import FusedConfig, quantize_activation, quantize_weight

    g = _gen(11)
    x = torch.randn(384, 512, device="cuda", generator=g)
    w = torch.randn(640, 512, device="cuda", generator=g) * 512 ** -0.5
    a, b = (quantize_activation(x), quantize_weight(w)) if fp8 else (x.to(torch.bfloat16), w.to(torch.bfloat16).t())
    ref = a.dequantize().double() @ b.dequantize().double() if fp8 else a.double() @ b.double()
    out = ctx.zeros((384, 640), dtype=torch.bfloat16)
    for variant in ("two_shot", "one_shot", "atomic") if op == "matmul_all_reduce" else ("auto",):
        for own in (True, False):
            ws = None
            for _ in range(3 if own else 1):
                out.zero_()
                ws = getattr(ctx.ops, op)(out, a, b, workspace=ws, config=FusedConfig(one_rank_fused=own, all_reduce_variant=variant), **kw)
                assert ws.variant == "fused" and bool(ws.extra["one_rank_fused"]) == own
                assert ((out.double() - ref).abs() <= 1.01 * 2.0 ** -8 * ref.abs() + 1e-4).all()
            assert own or (ws.inbox is None and ws.flags is None and ws.staging is None)
    ctx.check()


@pytest.mark.parametrize("config", [{}, {"block_size_n": 128}, {"block_size_n": 100}, {"two_sm": False}, {"two_sm": True}])
def test_one_rank_op_keeps_the_tile_it_is_asked_for(ctx, config):
    """128 rows go to the few-row kernel unless the config names a tile (100 is none of the kernel's widths: the plan's choice), also when
    only the workspace was made with it."""
    import ctypes as C

    from iris_b200 import _lib
    from iris_b200.ops import FusedConfig, all_gather_matmul_preamble

    cfg = FusedConfig(**config)
    asked = bool(config) and config.get("block_size_n") != 100
    g = _gen(9)
    x = torch.randn(128, 2048, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(1024, 2048, device="cuda", generator=g) * 2048 ** -0.5).to(torch.bfloat16).t()
    want = x.double() @ w.double()
    mark = ctx.heap_mark()
    for first, then in ((cfg, cfg), (cfg, None)):
        out = torch.empty(128, 1024, device="cuda", dtype=torch.bfloat16)
        ws = all_gather_matmul_preamble(ctx, x, w, first, shard_dim=0)
        ctx.ops.all_gather_matmul(out, x, w, shard_dim=0, config=first, workspace=ws)
        ctx.ops.all_gather_matmul(out, x, w, shard_dim=0, config=then, workspace=ws)
        (d, _), = ws.extra["desc"].values()
        assert ws.variant == "fused" and bool(_lib.kernels().iris_gemm_skinny_takes(C.byref(d))) == (not asked)
        assert ((out.double() - want).abs() <= 1.01 * 2.0 ** -8 * want.abs() + 1e-4).all()
    ctx.heap_release(mark)


@pytest.mark.parametrize("M,N,K", [(16, 3584, 512), (256, 4096, 2816), (300, 1000, 256), (2048, 2048, 64)])
def test_bias_inside_the_output(M, N, K):
    """A bias that is a row or a column of the output is read before the output is written: same bits as with a copy of it."""
    from iris_b200.ops import matmul

    g = _gen(M + N)
    A = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    B = (torch.randn(K, N, device="cuda", generator=g) * K ** -0.5).to(torch.bfloat16)
    out0 = torch.randn(M, N, device="cuda", generator=g).to(torch.bfloat16)
    for dim, pick in ((1, lambda t: t[0]), (1, lambda t: t[M - 1]), (0, lambda t: t[:, N - 1]), (0, lambda t: t[:, 0])):
        for _ in range(3):
            out = out0.clone()
            want = matmul(A, B, bias=pick(out).clone(), bias_dim=dim)
            assert torch.equal(matmul(A, B, bias=pick(out), bias_dim=dim, out=out), want)


def test_one_rank_op_broadcasts_one_row(ctx):
    """The result of one token is copied into an output of several rows, as by ``copy_``."""
    g = _gen(5)
    x = torch.randn(1, 256, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(256, 128, device="cuda", generator=g) * 256 ** -0.5).to(torch.bfloat16)
    out = torch.zeros(5, 128, device="cuda", dtype=torch.bfloat16)
    ctx.ops.all_gather_matmul(out, x, w, shard_dim=0)
    want = (x.double() @ w.double()).expand(5, 128)
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all()


def test_quantiser_special_values():
    """Infinities saturate, NaN counts as -448 and does not move its block's scale, zeros stay zero, in every position of
    a lane and of a block."""
    from iris_b200.ops.gemm_fp8 import quantize_activation

    for dtype in (torch.bfloat16, torch.float16, torch.float32):
        for pos in (0, 1, 7, 8, 63, 127):
            x = torch.ones(3, 256, device="cuda", dtype=dtype)
            x[0, pos], x[1, 128 + pos], x[2, :128] = float("nan"), float("inf"), 0.0
            got = quantize_activation(x)
            q = got.q.float()
            assert q[0, pos].item() == -448.0 and got.scale[0, 0].item() == got.scale[0, 1].item() == 2.0 ** -8
            assert q[1, 128 + pos].item() == 448.0 and got.scale[1, 1].item() == 2.0 ** 127
            assert (q[2, :128] == 0).all() and (q[2, 128:] == 256).all()


@pytest.mark.parametrize("S,Hq,Hkv", [(256, 2, 2), (768, 4, 2), (2560, 16, 2), (2560, 9, 3), (2816, 9, 3), (4352, 9, 3)])
@pytest.mark.parametrize("causal", [False, True])
def test_attention_zigzag_forms(ctx, S, Hq, Hkv, causal):
    """The zigzag walk (on one rank: plain attention) with a query tile's keys shared between the places, with two heads per item
    ((2560, 16, 2)), with neighbouring tiles of one head, and with a pair of them that lies in both halves of the block
    ((2816, 9, 3), 11 tiles each, full attention; (4352, 9, 3), 17 tiles each, causal too). Bounds as above."""
    from iris_b200.models import RingAttention, reference_attention

    g = _gen(S + Hq)
    mk = lambda h: torch.randn(S, h, 128, device="cuda", generator=g).clamp(-6, 6).to(torch.bfloat16)  # noqa: E731
    q, k, v = mk(Hq), mk(Hkv), mk(Hkv)
    mark = ctx.heap_mark()
    layer = RingAttention(ctx, S, Hq, Hkv, layout="zigzag")
    out = layer(q, k, v, causal=causal)
    assert (out.float() - reference_attention(q, k, v, causal)).abs().max().item() <= 2 * 2.0 ** -8 * 6
    assert torch.equal(out, layer(q, k, v, causal=causal))
    ctx.heap_release(mark)


@pytest.mark.parametrize("S,Hq,Hkv", [(384, 8, 8), (2500, 16, 8)])
def test_attention_largest_weight_is_exact(ctx, S, Hq, Hkv):
    """A row's largest weight is 1 before it is rounded to 16 bits, also when its key comes after the row's first tile (one
    of the first eight): key 300 outweighs the others by 2^0.3 to 2^7.3, at points between two bf16 values, and alone has a value, so
    that the output's own rounding (at most 2^-8 of it: bf16 has 8 significant bits) is all the error there is besides fp32's."""
    from iris_b200.models import RingAttention

    g = _gen(S)
    q = torch.ones(S, Hq, 128, device="cuda", dtype=torch.bfloat16)
    k, v = (torch.zeros(S, Hkv, 128, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    mark = ctx.heap_mark()
    layer = RingAttention(ctx, S, Hq, Hkv)
    for lo in (0.02, 0.15, 0.3):
        c = (lo + 0.15 * torch.rand(Hkv, device="cuda", generator=g)).to(torch.bfloat16)
        k[300] = c[:, None]
        v[300] = torch.randn(Hkv, 128, device="cuda", generator=g).to(torch.bfloat16)
        e = torch.exp(128 * c.double() * 128 ** -0.5)
        want = ((e / (e + S - 1))[:, None] * v[300].double()).repeat_interleave(Hq // Hkv, dim=0)
        assert ((layer(q, k, v).double() - want).abs() <= 1.01 * 2.0 ** -8 * want.abs()).all()
    ctx.heap_release(mark)


@pytest.mark.parametrize("S,layout", [(300, "contiguous"), (384, "contiguous"), (512, "zigzag")])
@pytest.mark.parametrize("sm_scale", [0.0, -0.05])
@pytest.mark.parametrize("causal", [False, True])
def test_attention_scale_that_is_not_positive(ctx, S, layout, sm_scale, causal):
    """Masked keys stay masked and the maximum stays a maximum: 0 weighs every key that a row sees alike, a negative scale
    prefers the lowest products. Same bound as above (|v| < 6)."""
    from iris_b200.models import RingAttention, reference_attention

    g = _gen(S)
    q, k, v = (torch.randn(S, 4, 128, device="cuda", generator=g).clamp(-6, 6).to(torch.bfloat16) for _ in range(3))
    mark = ctx.heap_mark()
    out = RingAttention(ctx, S, 4, 4, sm_scale=sm_scale, layout=layout)(q, k, v, causal=causal)
    assert (out.float() - reference_attention(q, k, v, causal, sm_scale=sm_scale)).abs().max().item() <= 2 * 2.0 ** -8 * 6
    ctx.heap_release(mark)


@pytest.mark.parametrize("S", [300, 384])
@pytest.mark.parametrize("tc", [None, False])
def test_attention_rows_whose_first_keys_score_minus_infinity(ctx, S, tc):
    """Keys with -inf in a column where every query is 1 score -inf: whole tiles of them in front of the others change
    nothing, and a row that sees only such keys has weight 0 and a log-sum of -inf."""
    from iris_b200.models import RingAttention, reference_attention

    g = _gen(S)
    q, k, v = (torch.randn(S, 4, 128, device="cuda", generator=g).clamp(-6, 6).to(torch.bfloat16) for _ in range(3))
    q[..., 0], k[..., 0], k[:200, :, 0] = 1.0, 0.0, float("-inf")
    mark = ctx.heap_mark()
    layer = RingAttention(ctx, S, 4, 4, use_tcgen05=tc)
    for causal in (False, True):
        out, lse = layer(q, k, v, causal=causal, return_lse=True)
        want = reference_attention(q, k[200:], v[200:], causal, q_offset=-200) if causal else reference_attention(q, k[200:], v[200:])
        first = 200 if causal else 0
        assert (out[first:].float() - want[first:]).abs().max().item() <= 2 * 2.0 ** -8 * 6
        assert (out[:first] == 0).all() and torch.isneginf(lse[:first]).all() and torch.isfinite(lse[first:]).all()
    ctx.heap_release(mark)
