"""FP8 weights with a scale per output channel: the one-launch packer against the scalar definition, over rows of one
vector, rows past what a block holds, and the forms that keep the general kernels (odd K, an unaligned source)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("source_type", [torch.float16, torch.float32])
@pytest.mark.parametrize("name", ["e4m3", "e5m2"])
@pytest.mark.parametrize("n,k,offset", [(1, 8, 0), (3, 1024, 0), (17, 1032, 0), (5, 5120, 0), (4, 5128, 0), (2, 10248, 0), (6, 639, 0), (4, 640, 1)])
def test_packed_rows(gpu, source_type, name, n, k, offset):
    pkg, ctx, ops = gpu
    torch.manual_seed(k)
    source = torch.randn(n * k + offset, device="cuda").to(source_type)[offset:].view(n, k)
    source[0, k // 2] = float("inf")                                   # the scale is taken over finite values
    if n > 2:
        source[2] = 0.0
    dtype, most = {"e4m3": (torch.float8_e4m3fn, 448.0), "e5m2": (torch.float8_e5m2, 57344.0)}[name]
    fmt = {"e4m3": pkg.ScalarType.Float8E4M3, "e5m2": pkg.ScalarType.Float8E5M2}[name]
    w = ops.upload_fp8_weight(source, pkg.FP8WeightLoadOptions(format=fmt, scale_mode=pkg.FP8ScaleMode.PerOutputChannel))
    ctx.check()
    values = source.float()
    amax = torch.where(values.isfinite(), values.abs(), torch.zeros_like(values)).amax(dim=1)
    scale = torch.where(amax > 0, torch.clamp(amax / torch.full_like(amax, most), min=1e-12), torch.ones_like(amax))
    want = (values / scale[:, None]).clamp(-most, most).to(dtype).view(torch.uint8)
    assert torch.equal(w.scales, scale)
    assert torch.equal(w.data.view(torch.uint8).view(n, k), want)
