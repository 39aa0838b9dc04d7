"""The epilogue forms that run ahead of the accumulators or evaluate a chunk's values together: residual loads in a
ring of four chunks per warp, and the activation of 16 values at once."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def packed(pkg, ops, dtype, n, k):
    source = (torch.randn(n, k, device="cuda") / k ** 0.5).half()
    if dtype == "int8":
        return ops.upload_or_quantize_int8_weight(source, None, pkg.INT8WeightLoadOptions(enable_convrot=False))
    if dtype == "e4m3":
        return ops.upload_fp8_weight(source, pkg.FP8WeightLoadOptions(scale_mode=pkg.FP8ScaleMode.PerOutputChannel))
    return ops.fp16_weight(source)


@pytest.mark.parametrize("dtype", ["int8", "e4m3", "f16"])
@pytest.mark.parametrize("pair", [0, 1])
@pytest.mark.parametrize("m,n,tile_n", [(1, 16, 16), (130, 40, 48), (257, 136, 144), (300, 264, 256), (128, 520, 256), (513, 1288, 160)])
def test_residual_is_added_to_the_projection(gpu, dtype, pair, m, n, tile_n):
    """half(projection + bias) + residual in one rounding more, element for element: bit-equal to the projection
    without it followed by an FP16 addition, with the residual apart from and aliased to the output."""
    pkg, ctx, ops = gpu
    torch.manual_seed(m + n)
    k = 192
    weight = packed(pkg, ops, dtype, n, k)
    x, residual = torch.randn(m, k, device="cuda").half(), torch.randn(m, n, device="cuda").half()
    bias = torch.randn(n, device="cuda").half()
    ctx.set_pair_mode(pair)
    ctx.set_tile_n(tile_n)
    want = ops.linear(x, weight, bias) + residual
    assert torch.equal(ops.linear(x, weight, bias, residual=residual), want)
    amax = torch.zeros(1, dtype=torch.int32, device="cuda")
    in_place = residual.clone()
    ops.linear(x, weight, bias, residual=in_place, out=in_place, y_amax=amax)
    assert torch.equal(in_place, want)
    assert amax.view(torch.float32).item() == want.abs().max().float().item()
    ctx.check()
