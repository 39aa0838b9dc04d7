"""The native front (csrc/torch_front.cpp) and the ctypes path issue the same calls: same bits for every form
of argument, and the front hands over what it does not take, so that errors keep their messages."""
import pytest
import torch

import helpers

pytestmark = pytest.mark.gpu


class _NoFront:
    """Answers None to everything: the Python path runs."""

    def __getattr__(self, name):
        return lambda *arguments: None


@pytest.mark.parametrize("dtype", ["int8", "e4m3", "f16"])
@pytest.mark.parametrize("lead", [(5,), (2, 77), (1, 3, 7)])
def test_front_and_python_path_agree(gpu, dtype, lead):
    pkg, ctx, ops = gpu
    slow = pkg.Ops(ctx, poison_outputs=True)
    slow._front = _NoFront()
    torch.manual_seed(3)
    k, n = 256, 64
    x = torch.randn(*lead, k, device="cuda").half()
    source = (torch.randn(n, k, device="cuda") / 16).half()
    bias, gamma, beta = torch.randn(n, device="cuda").half(), torch.rand(k, device="cuda").half(), torch.randn(k, device="cuda").half()
    residual = torch.randn(*lead, n, device="cuda").half()
    results = []
    for o in (ops, slow):
        if dtype == "int8":
            w = o.upload_or_quantize_int8_weight(source, None, pkg.INT8WeightLoadOptions())
            q = o.quantize_int8(x, 256)
        elif dtype == "e4m3":
            w = o.upload_fp8_weight(source, pkg.FP8WeightLoadOptions(scale_mode=pkg.FP8ScaleMode.PerOutputChannel))
            quantised = o.quantize_e4m3(x)
            q = (quantised.data, quantised.scales)
        else:
            w, q = o.fp16_weight(source), ()
        out = [w.data, *([w.scales] if w.scales is not None else []), *q]
        out += [o.linear(x, w), o.linear(x, w, bias, residual=residual), o.linear_activation(x, w, bias, pkg.ACT_GEGLU)]
        calls = [pkg.LinearCall(x, w), pkg.LinearCall(x, w, bias, pkg.ACT_SILU)]
        out += o.linear_grouped(calls)
        assert calls[1].y is out[-1]
        out.append(o.layer_norm(x, gamma, beta))
        if dtype != "f16":
            pair = o.layer_norm_quantized(x, gamma, beta, w)
            out += [*pair, o.linear(None, w, bias, xq=pair[0], xq_scales=pair[1])]
        results.append(out)
    ctx.check()
    for fast, plain in zip(*results):
        assert fast.shape == plain.shape and fast.dtype == plain.dtype and torch.equal(fast, plain)


def test_front_leaves_errors_to_the_python_path(gpu):
    pkg, ctx, ops = gpu
    w = ops.fp16_weight(torch.zeros(64, 32, device="cuda"))
    with pytest.raises(pkg.CudaError, match="contiguous"):
        ops.linear(torch.zeros(32, 8, device="cuda", dtype=torch.float16).t(), w)
    with pytest.raises(pkg.CudaError, match="feature mismatch"):
        ops.linear(torch.zeros(8, 16, device="cuda", dtype=torch.float16), w)
    with pytest.raises(pkg.CudaError, match="requires a bias"):         # found by the library behind the front
        ops.linear_activation(torch.zeros(8, 32, device="cuda", dtype=torch.float16), w, None, pkg.ACT_SILU)


def test_outputs_that_share_copy_on_write_storage(gpu):
    """A tensor the call writes gets its own memory; the tensor it was lazily cloned from keeps its values."""
    pkg, ctx, ops = gpu
    torch.manual_seed(4)
    weight = ops.upload_or_quantize_int8_weight(torch.randn(64, 64, device="cuda"), None, pkg.INT8WeightLoadOptions(enable_convrot=False))
    fp8 = ops.upload_fp8_weight(torch.randn(64, 64, device="cuda"), pkg.FP8WeightLoadOptions())
    x, ones = torch.randn(20, 64, device="cuda").half(), torch.ones(64, device="cuda").half()
    kept = {"y": torch.full((20, 64), 3.0, device="cuda", dtype=torch.float16), "acc": torch.full((20, 64), 3, device="cuda", dtype=torch.int32),
            "amax": torch.zeros(1, device="cuda", dtype=torch.int32)}
    before = {name: t.clone() for name, t in kept.items()}
    clones = [{name: torch._lazy_clone(t) for name, t in kept.items()} for _ in range(4)]
    assert ops.linear(x, weight, out=clones[0]["y"], acc_out=clones[0]["acc"], y_amax=clones[0]["amax"]) is clones[0]["y"]
    ops.linear_grouped([pkg.LinearCall(x, weight, y=clones[1]["y"])])
    ops.layer_norm(x, ones, ones, out=clones[2]["y"])
    assert clones[0]["amax"].item() != 0 and not torch.equal(clones[0]["acc"], before["acc"])
    word = clones[0]["amax"]
    shared = torch._lazy_clone(word)
    left = shared.item()
    ops.linear(clones[0]["y"], fp8, x_amax=word)                   # reads the word and puts it back to zero
    ctx.check()
    assert word.item() == 0 and shared.item() == left
    assert not any(torch.equal(clones[i]["y"], before["y"]) for i in range(3))
    for name, t in kept.items():
        assert torch.equal(t, before[name])


def test_outputs_are_allocated_through_the_dispatcher(gpu):
    """A dispatch mode sees the allocations, and deterministic mode fills them, as on the Python path."""
    from torch.utils._python_dispatch import TorchDispatchMode
    pkg, ctx, ops = gpu
    weight = ops.fp16_weight(torch.randn(64, 64, device="cuda").half())
    x, ones = torch.randn(4, 64, device="cuda").half(), torch.ones(64, device="cuda").half()

    class Record(TorchDispatchMode):
        seen = 0

        def __torch_dispatch__(self, function, types, args=(), kwargs=None):
            Record.seen += "empty" in str(function)
            return function(*args, **(kwargs or {}))

    plain = pkg.Ops(ctx)
    with Record():
        plain.linear(x, weight)
        plain.linear_grouped([pkg.LinearCall(x, weight), pkg.LinearCall(x, weight)])
        plain.layer_norm(x, ones, ones)
        plain.quantize_int8(x, 0)
        plain.quantize_e4m3(x)
    assert Record.seen == 1 + 2 + 1 + 2 + 2

    assert not any("Fill" in kernel.name for kernel in helpers.launches(ctx, lambda: plain.linear(x, weight)))
    torch.use_deterministic_algorithms(True)
    try:
        kernels = helpers.launches(ctx, lambda: plain.linear(x, weight))
    finally:
        torch.use_deterministic_algorithms(False)
    assert any("Fill" in kernel.name for kernel in kernels)
    ctx.check()


@pytest.mark.parametrize("missing", ["bias", "residual", "acc_out", "y", "x_amax"])
def test_front_leaves_incomplete_objects_to_the_python_path(gpu, missing):
    """An attribute that does not exist is not None."""
    from types import SimpleNamespace
    pkg, ctx, ops = gpu
    weight = ops.fp16_weight(torch.zeros(64, 32, device="cuda"))
    call = vars(pkg.LinearCall(torch.zeros(4, 32, device="cuda").half(), weight))
    with pytest.raises(AttributeError):
        ops.linear_grouped([SimpleNamespace(**{name: value for name, value in call.items() if name != missing})])
    with pytest.raises(AttributeError):
        ops.linear(call["x"], SimpleNamespace(**{name: value for name, value in vars(weight).items() if name != "scales"}))
