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
