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
