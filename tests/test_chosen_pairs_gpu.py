"""Shapes for which single calls take CTA pairs by themselves (GEGLU of many tiles, a long K with few), at and beside
the rule's edges: the results equal those of single CTAs bit for bit in every type (the MMAs of a pair add the same
products in the same order), with every output and epilogue a call can ask for."""
import pytest
import torch

import helpers

pytestmark = pytest.mark.gpu


def pack(pkg, ops, dtype, source):
    if dtype.startswith("int8"):
        group = int(dtype[4:] or 0)
        return ops.upload_or_quantize_int8_weight(source, None, pkg.INT8WeightLoadOptions(enable_convrot=group != 0, convrot_group_size=group))
    if dtype == "f16":
        return ops.fp16_weight(source)
    fmt = {"e4m3": pkg.ScalarType.Float8E4M3, "e5m2": pkg.ScalarType.Float8E5M2}[dtype]
    return ops.upload_fp8_weight(source, pkg.FP8WeightLoadOptions(format=fmt, scale_mode=pkg.FP8ScaleMode.PerOutputChannel))


@pytest.mark.parametrize("dtype", ["int8", "int816", "e4m3", "e5m2", "f16"])
@pytest.mark.parametrize("m,n,k,geglu", [(129, 64, 4096, False), (154, 1280, 5120, False), (257, 648, 4112, False), (2048, 1280, 3968, False), (4097, 640, 2560, False),
                                         (1976, 1280, 5120, False), (128, 1280, 5120, False), (3000, 5120, 640, True), (8192, 5120, 128, True),
                                         (1976, 10240, 1280, True)])
def test_same_bits_as_single_ctas(pkg, gpu_session, dtype, m, n, k, geglu):
    _, _, reference = gpu_session
    reference.ctx.set_pair_mode(0)
    reference.ctx.set_tile_n(0)
    context = pkg.Context(0, workspace_bytes=256 << 20)
    ops = pkg.Ops(context, poison_outputs=True)
    torch.manual_seed(m)
    weight = pack(pkg, ops, dtype, (torch.randn(n, k, device="cuda") / k ** 0.5).half())
    x, bias = torch.randn(m, k, device="cuda").half(), torch.randn(n, device="cuda").half()
    for o in (ops, reference):
        amax = torch.zeros(1, dtype=torch.int32, device="cuda")
        if geglu:
            o.result = [o.linear_activation(x, weight, bias, pkg.ACT_GEGLU, y_amax=amax), amax]
        else:
            residual = torch.randn(m, n, device="cuda", generator=torch.Generator("cuda").manual_seed(1)).half()
            o.result = [o.linear(x, weight, bias), o.linear(x, weight, bias, residual=residual, y_amax=amax), amax]
            o.result += [o.linear_activation(x, weight, bias, activation) for activation in (pkg.ACT_SILU, pkg.ACT_GELU, pkg.ACT_QUICK_GELU)]
            o.result += o.linear_grouped([pkg.LinearCall(x, weight), pkg.LinearCall(x, weight, bias)])
            if dtype.startswith("int8"):
                accumulators = torch.zeros(m, n, dtype=torch.int32, device="cuda")
                o.result += [o.linear(x, weight, acc_out=accumulators), accumulators]
    context.check()
    for got, want in zip(ops.result, reference.result):
        assert torch.equal(got, want)
    context.close()


@pytest.mark.parametrize("m,n,k,activation,pairs", [
    (128, 1280, 5120, "none", ""), (129, 1280, 5120, "none", "int8 e4m3 f16"), (300, 1280, 4096, "silu", "int8 e4m3 f16"),
    (300, 1280, 3968, "none", "f16"), (300, 1280, 1984, "none", ""), (3000, 1280, 5120, "none", "f16"), (4000, 1280, 5120, "gelu", "int8 e4m3 f16"),
    (5000, 640, 2560, "none", ""), (7000, 640, 2560, "none", "int8 e4m3 f16"), (3000, 1280, 4032, "none", ""), (7000, 640, 2432, "none", "f16"), (4736, 640, 8192, "none", ""), (8192, 640, 1216, "none", ""),
    (1000, 5120, 640, "geglu", ""), (8192, 5120, 640, "geglu", "int8 e4m3 f16"), (65536, 640, 2560, "none", "")])
def test_which_calls_take_pairs(pkg, gpu_session, m, n, k, activation, pairs):
    """Both sides of the rule's lines, for a context whose pair mode was never set."""
    context = pkg.Context(0, workspace_bytes=256 << 20)
    ops = pkg.Ops(context)
    x, bias = torch.zeros(m, k, device="cuda").half(), torch.zeros(n, device="cuda").half()
    kinds = {"none": None, "silu": pkg.ACT_SILU, "gelu": pkg.ACT_GELU, "geglu": pkg.ACT_GEGLU}
    for dtype in ("int8", "e4m3", "f16"):
        weight = pack(pkg, ops, dtype, torch.ones(n, k, device="cuda").half())

        def call():
            return ops.linear(x, weight, bias) if activation == "none" else ops.linear_activation(x, weight, bias, kinds[activation])
        gemms = [kernel for kernel in helpers.launches(context, call) if "umma_gemm" in kernel.name]
        assert len(gemms) == 1 and (gemms[0].cluster == 2) == (dtype in pairs.split())
    context.check()
    context.close()


@pytest.mark.parametrize("dtype", ["int8", "e4m3", "f16"])
@pytest.mark.parametrize("shapes", [[(154, 1280, 1280), (154, 1280, 4096)], [(2048, 1280, 1280), (154, 1280, 4096), (154, 1280, 4096)],
                                    [(300, 1280, 5120), (300, 1280, 64)], [(257, 648, 5120), (300, 1280, 5120)]])
def test_a_small_group_is_one_launch(pkg, gpu_session, dtype, shapes):
    """Members with and without pairs by the rule (a long K beside a short one), or all with pairs: one GEMM launch, and
    the bits of the single calls."""
    context = pkg.Context(0, workspace_bytes=256 << 20)
    ops = pkg.Ops(context, poison_outputs=True)
    torch.manual_seed(1)
    calls = []
    for m, n, k in shapes:
        weight = pack(pkg, ops, dtype, (torch.randn(n, k, device="cuda") / k ** 0.5).half())
        x = torch.randn(m, k, device="cuda").half()
        given = {}
        if dtype == "int8":
            given = dict(zip(("xq", "xq_scales"), ops.quantize_int8(x, 0)))
        elif dtype == "e4m3":
            cast = ops.quantize_e4m3(x)
            given = {"xq": cast.data, "xq_scales": cast.scales}
        calls.append((x, weight, given))
    def group():
        return ops.linear_grouped([pkg.LinearCall(x, w, **given) for x, w, given in calls])

    assert sum("umma_gemm" in kernel.name for kernel in helpers.launches(context, group)) == 1
    for got, (x, weight, given) in zip(group(), calls):
        assert torch.equal(got, ops.linear(x, weight, **given))
    context.check()
    context.close()


def test_the_default_choice_can_be_set_again(pkg, gpu):
    _, context, ops = gpu
    x = torch.zeros(300, 5120, device="cuda").half()
    weights = [ops.fp16_weight(torch.zeros(1280, k, device="cuda")) for k in (5120, 64)]
    inputs = [x, x[:, :64].contiguous()]

    def pairs():
        kernels = helpers.launches(context, lambda: [ops.linear(a, w) for a, w in zip(inputs, weights)])
        return sorted(kernel.cluster for kernel in kernels if "umma_gemm" in kernel.name)

    assert pairs() == [1, 2]
    for mode, want in ((0, [1, 1]), (1, [2, 2]), (-1, [1, 1]), (2, [1, 2])):
        context.set_pair_mode(mode)
        assert pairs() == want
    for mode in (-2, 3):
        with pytest.raises(pkg.CudaError):
            context.set_pair_mode(mode)
    assert pairs() == [1, 2]
