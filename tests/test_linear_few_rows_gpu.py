"""Projections of at most 16 rows (csrc/linear_skinny.cu) against the tensor-memory GEMM, which a forced tile width
brings back: INT8 bit-equal. FP8 and FP16 sum in another order: K / 16 MMA steps, each off by at most 2^-23 of a partial
sum no larger than the sum S of the products' magnitudes, then the FP16 rounding of the projection may fall the other way."""
import pytest
import torch

import helpers

pytestmark = pytest.mark.gpu


def matrix(n, k):
    return (torch.randn(n, k, device="cuda") / k ** 0.5).half()


def make(pkg, ops, dtype, n, k, source):
    if dtype.startswith("int8"):
        group = int(dtype[4:] or 0)
        return ops.upload_or_quantize_int8_weight(source, None, pkg.INT8WeightLoadOptions(enable_convrot=group != 0, convrot_group_size=group))
    if dtype == "f16":
        return ops.fp16_weight(source)
    fmt = {"e4m3": pkg.ScalarType.Float8E4M3, "e5m2": pkg.ScalarType.Float8E5M2}[dtype]
    mode = pkg.FP8ScaleMode.PerOutputChannel if k % 32 else pkg.FP8ScaleMode.TensorWide
    return ops.upload_fp8_weight(source, pkg.FP8WeightLoadOptions(format=fmt, scale_mode=mode))


def agree(got, want, exact, bound):
    if exact:
        assert torch.equal(got, want)
    else:
        assert ((got.float() - want.float()).abs() <= bound + want.abs().float() * 2.0 ** -10).all()


@pytest.mark.parametrize("dtype", ["int8", "int864", "int8256", "e4m3", "e5m2", "f16"])
@pytest.mark.parametrize("m,n,k", [(1, 16, 256), (2, 1280, 320), (7, 24, 1040), (8, 2600, 64), (9, 5200, 512), (16, 1280, 2816), (16, 40, 5120), (13, 8, 16)])
def test_against_the_tensor_memory_gemm(gpu, dtype, m, n, k):
    pkg, ctx, ops = gpu
    if dtype.startswith("int8") and k % int(dtype[4:] or 1):
        pytest.skip("the group size does not divide K")
    torch.manual_seed(n + k)
    source = matrix(n, k)
    weight = make(pkg, ops, dtype, n, k, source)
    x = torch.randn(m, k, device="cuda").half()
    x[:, :: max(1, k // 3)] *= 20
    bias, residual = torch.randn(n, device="cuda").half(), torch.randn(m, n, device="cuda").half()
    amax = torch.zeros(2, dtype=torch.int32, device="cuda")
    results = []
    for tile in (0, 32):
        ctx.set_tile_n(tile)
        out = [ops.linear(x, weight), ops.linear(x, weight, bias, residual=residual, y_amax=amax[tile // 32:][:1])]
        out += [ops.linear_activation(x, weight, bias, a) for a in (pkg.ACT_SILU, pkg.ACT_GELU, pkg.ACT_QUICK_GELU, pkg.ACT_GEGLU)]
        if dtype.startswith("int8"):
            accumulators = torch.zeros(m, n, dtype=torch.int32, device="cuda")
            ops.linear(x, weight, acc_out=accumulators)
            out.append(accumulators)
        results.append(out)
    ctx.set_tile_n(0)
    ctx.check()
    projection = results[1][0].abs().float()
    magnitudes = 1.2 * x.abs().float() @ source.abs().float().T          # 1.2: quantised values are up to an eighth larger
    off = projection * 2.0 ** -10 + k / 16 * 2.0 ** -23 * magnitudes     # of the projection
    half = n // 2
    value, gate = projection[:, :half] + 5.0, projection[:, half:] + 5.0     # with their bias
    bounds = [off, off] + [1.2 * off] * 3 + [off[:, :half] * gate + 1.2 * value * off[:, half:]]      # activations' slope: < 1.2
    for at, (got, want) in enumerate(zip(*results)):
        agree(got, want, dtype.startswith("int8"), bounds[at] if at < 6 else None)
    assert amax[:1].view(torch.float32).item() == results[0][1].abs().max().float().item()


@pytest.mark.parametrize("dtype", ["int8", "e4m3", "e5m2"])
@pytest.mark.parametrize("m,k", [(1, 64), (2, 1280), (16, 2816), (16, 8208)])
def test_own_quantisation_is_the_quantisers(gpu, dtype, m, k):
    """FP16 input and input cast by the stand-alone quantiser give the same bits (also past the size at which the kernel
    quantises for itself), for rows of zeros, infinities (INT8: the finite maximum) and tiny values too."""
    pkg, ctx, ops = gpu
    torch.manual_seed(k)
    weight = make(pkg, ops, dtype, 96, k, matrix(96, k))
    x = torch.randn(m, k, device="cuda").half()
    if m > 2:
        x[1], x[2] = 0.0, x[2] * 1e-7
        if dtype == "int8":
            x[3, 5] = float("inf")
    if dtype == "int8":
        xq, scales = ops.quantize_int8(x, 0)
    else:
        quantised = ops.quantize_fp8(x, weight.type)
        xq, scales = quantised.data, quantised.scales
    assert torch.equal(ops.linear(x, weight), ops.linear(None, weight, xq=xq, xq_scales=scales))
    ctx.check()


@pytest.mark.parametrize("dtype", ["int8", "int8256", "e4m3", "e5m2"])
@pytest.mark.parametrize("m,k,shift", [(2, 64, 0), (16, 1280, 0), (16, 1280, 640), (16, 5120, 0)])
def test_projection_in_place(gpu, dtype, m, k, shift):
    """A square projection written over its own input (or half a row behind it): the input is read whole before the first
    store, also where the grid takes more than one wave of blocks ([16, 5120])."""
    pkg, ctx, ops = gpu
    if dtype == "int8256" and k % 256:
        pytest.skip("the group size does not divide K")
    torch.manual_seed(k)
    weight = make(pkg, ops, dtype, k, k, matrix(k, k))
    bias, values = torch.randn(k, device="cuda").half(), torch.randn(m, k, device="cuda").half()
    want = ops.linear(values, weight, bias, residual=values)
    for with_residual in (False, True) if shift == 0 else (False,):
        buffer = torch.zeros(m * k + shift, device="cuda", dtype=torch.float16)
        x, out = buffer[:m * k].view(m, k), buffer[shift:].view(m, k)
        x.copy_(values)
        ops.linear(x, weight, bias, residual=x if with_residual else None, out=out)
        assert torch.equal(out, want if with_residual else ops.linear(values, weight, bias))
    ctx.check()


@pytest.mark.parametrize("dtype,m,n,k,activation,expected", [
    ("f16", 16, 4736, 64, "none", "skinny"), ("f16", 16, 5120, 64, "none", "skinny"), ("f16", 17, 64, 64, "none", "gemm"),
    ("f16", 8, 10240, 64, "none", "skinny"), ("f16", 9, 10240, 64, "none", "gemm"), ("f16", 16, 10240, 64, "geglu", "skinny"), ("f16", 1, 20480, 64, "none", "gemm"),
    ("int8", 16, 4736, 1280, "none", "skinny"), ("int8", 12, 5120, 64, "none", "skinny"), ("int8", 13, 5120, 64, "none", "quantiser gemm"),
    ("int8", 2, 9504, 64, "none", "quantiser skinny"), ("int8", 16, 64, 1296, "none", "quantiser skinny"), ("int8256", 6, 10240, 256, "none", "quantiser skinny"),
    ("int8256", 7, 10240, 256, "none", "quantiser gemm"), ("e4m3", 16, 4736, 64, "none", "skinny"), ("e4m3", 12, 5120, 64, "none", "skinny"),
    ("e5m2", 13, 5120, 64, "none", "quantiser quantiser gemm"), ("e4m3", 1, 9504, 64, "none", "quantiser quantiser gemm"), ("e4m3", 16, 64, 8208, "none", "quantiser quantiser skinny"),
    ("e4m3", 16, 64, 8192, "none", "skinny"), ("e4m3", 8, 10240, 64, "geglu", "quantiser quantiser gemm")])
def test_which_calls_take_the_few_row_kernel(gpu, dtype, m, n, k, activation, expected):
    """Both sides of the rule's lines, on 148 SMs."""
    pkg, ctx, ops = gpu
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the sizes are those of 148 SMs")
    weight = make(pkg, ops, dtype, n, k, torch.ones(n, k, device="cuda").half())
    x, bias = torch.zeros(m, k, device="cuda").half(), torch.zeros(n, device="cuda").half()
    kernels = helpers.launches(ctx, lambda: ops.linear(x, weight, bias) if activation == "none" else ops.linear_activation(x, weight, bias, pkg.ACT_GEGLU))
    families = {"skinny": "skinny", "umma_gemm": "gemm", "fp8_amax": "quantiser", "fp8_cast": "quantiser", "plain_rows": "quantiser", "rotated": "quantiser"}
    found = [family for kernel in kernels for part, family in families.items() if part in kernel.name]
    assert sorted(found) == sorted(expected.split())
