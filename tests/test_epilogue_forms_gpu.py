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


@pytest.mark.parametrize("offset", [1, 8, 24])
@pytest.mark.parametrize("m", [3, 130])
def test_residual_with_an_alignment_of_its_own(gpu, offset, m):
    """A contiguous residual 2, 16 or 48 bytes into its buffer, beside an output that takes 32-byte accesses."""
    pkg, ctx, ops = gpu
    torch.manual_seed(offset)
    n, k = 48, 64
    weight = packed(pkg, ops, "f16", n, k)
    x, bias = torch.randn(m, k, device="cuda").half(), torch.randn(n, device="cuda").half()
    residual = torch.randn(m * n + offset, device="cuda").half()[offset:].view(m, n)
    assert torch.equal(ops.linear(x, weight, bias, residual=residual), ops.linear(x, weight, bias) + residual)
    ctx.check()


@pytest.mark.parametrize("name", ["silu", "gelu", "quick_gelu"])
@pytest.mark.parametrize("n", [16, 40, 264])
def test_activation_of_a_chunk(gpu, name, n):
    """act(half(projection) + bias) against 64 bits from the same halves, over the whole FP16 range of arguments. The
    FP32 evaluation is good to a few 2^-22 relative, and GELU's to |x| / 2 times the 6e-7 of its erfc, so its FP16 rounding
    is within that and one step of the exactly rounded one."""
    pkg, ctx, ops = gpu
    k = 64
    weight = ops.fp16_weight(torch.eye(n, k, device="cuda").half())
    values = torch.cat([torch.linspace(-12, 12, 4000), torch.tensor([0.0, -0.0, 65504.0, -65504.0, 88.0, -88.0, 104.0, -104.0, 6e-8, -6e-8]),
                        10.0 ** torch.linspace(-7, 4.8, 500), -(10.0 ** torch.linspace(-7, 4.8, 500))]).half()
    columns = min(n, k)
    m = -(-values.numel() // columns)
    x = torch.zeros(m * columns).half()
    x[:values.numel()] = values
    padded = torch.zeros(m, k).half()
    padded[:, :columns] = x.view(m, columns)
    activation = {"silu": pkg.ACT_SILU, "gelu": pkg.ACT_GELU, "quick_gelu": pkg.ACT_QUICK_GELU}[name]
    got = ops.linear_activation(padded.cuda(), weight, torch.zeros(n, device="cuda").half(), activation).cpu()
    ctx.check()
    z = torch.zeros(m, n, dtype=torch.float64)
    z[:, :columns] = padded[:, :columns].double()
    if name == "gelu":
        from scipy.special import erfc
        want = torch.from_numpy(0.5 * z.numpy() * erfc(-z.numpy() / np.sqrt(2.0)))
    else:
        want = z * torch.sigmoid(z * (1.0 if name == "silu" else 1.702))
    rounded = want.half()
    step = torch.maximum(rounded.double().abs() * 2.0 ** -10, torch.full_like(want, 2.0 ** -24))
    assert (got.double() - rounded.double()).abs().le(step + 3e-7 * z.abs() * (name == "gelu")).all()


@pytest.mark.parametrize("m,tile_n", [(3, 0), (3, 16), (17, 0), (130, 0)])
def test_activation_of_infinities_and_zeros(gpu, m, tile_n):
    """x / (1 + exp(-x)) as IEEE has it: +inf stays, -inf and NaN give NaN, a zero keeps its sign; on the few-row
    kernel (3 rows) and in the epilogue of the tensor-memory GEMM (a forced tile width, or more than 16 rows)."""
    pkg, ctx, ops = gpu
    ctx.set_tile_n(tile_n)
    weight = torch.eye(16, 64, device="cuda").half() * 2
    weight[1, 1] = 0.25
    weight = ops.fp16_weight(weight)
    bias = torch.zeros(16, device="cuda").half()
    bias[1] = -0.0
    x = torch.zeros(m, 64).half()
    last = m - 1
    x[last - 2, 0], x[last - 1, 0], x[last, 0] = 65504.0, -65504.0, float("nan")       # doubled: +-inf
    x[last - 2, 1] = -2.0 ** -24                                                      # a quarter of it rounds to -0
    for activation in (pkg.ACT_SILU, pkg.ACT_QUICK_GELU):
        y = ops.linear_activation(x.cuda(), weight, bias, activation).cpu()
        assert y[last - 2, 0] == float("inf") and torch.isnan(y[last - 1, 0]) and torch.isnan(y[last]).all()
        assert y[last - 2, 1] == 0 and torch.signbit(y[last - 2, 1]) and not torch.signbit(y[last - 2, 2])
    ctx.set_tile_n(0)
    ctx.check()
