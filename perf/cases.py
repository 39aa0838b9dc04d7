"""The work that users of the quantized-Linear path have it do, as cases that can be timed and compared.

Kinds of case, each through the package's public entry points on the GPU:
  linear       one projection: Ops.linear / Ops.linear_activation
  block        the norms and projections of one transformer block, in the order a UNet step runs them
               (the two attention results come from the caller)
  cross_kv     every cross-attention to_k / to_v of the UNet in one grouped plan, once per generation
  projections  all 743 projections of one UNet step as one grouped plan
  load         the weights of one transformer block packed from a checkpoint's FP16 / FP32 tensors
  denoise      one Euler step of the synthetic SDXL Base UNet loop, replayed as a CUDA graph

Row counts follow from an image size and a number of images with CFG (UNet batch = 2 x images): 64 x 64
latent tokens per 1024 x 1024 image at the 640-wide level, 32 x 32 at the 1280-wide one, 77 context tokens.
"""
import functools
import importlib
import math

import torch

pkg = importlib.import_module("sdxl-end2end_b200")
shapes = importlib.import_module("sdxl-end2end_b200.unet_shapes")

ACTIVATIONS = {"none": pkg.ACT_NONE, "silu": pkg.ACT_SILU, "gelu": pkg.ACT_GELU, "quick_gelu": pkg.ACT_QUICK_GELU,
               "geglu": pkg.ACT_GEGLU}
CONTEXT_TOKENS, CROSS_DIM = 77, 2048


def tokens(case, width):
    """Rows of the token matrices of a level for the case's images."""
    shrink = {640: 16, 1280: 32}[width]
    return 2 * case["images"] * (case["height"] // shrink) * (case["width"] // shrink)


def image(images, height=1024, width=1024):
    return {"images": images, "height": height, "width": width}


def listed():
    return [
        # time_embedding.linear_1 for one image: the smallest projection, all latency
        {"name": "time_embedding", "kind": "linear", "m": 2, "n": 1280, "k": 320, "dtype": "e4m3", "scales": "channel",
         "group": 0, "activation": "silu", "residual": False},
        # add_embedding.linear_1 for eight images: few rows, a long K, rotated INT8 rows
        {"name": "label_embedding", "kind": "linear", "m": 16, "n": 1280, "k": 2816, "dtype": "int8", "scales": "channel",
         "group": 256, "activation": "silu", "residual": False},
        # fc1 of the smaller text encoder for one prompt pair: ragged rows, FP16 weights
        {"name": "text_encoder_fc1", "kind": "linear", "m": 154, "n": 3072, "k": 768, "dtype": "f16", "scales": "none",
         "group": 0, "activation": "quick_gelu", "residual": False},
        # ff.net.0.proj of the 640-wide level with FP16 weights, one image at 1024 x 1024
        {"name": "geglu_f16", "kind": "linear", "m": 8192, "n": 5120, "k": 640, "dtype": "f16", "scales": "none",
         "group": 0, "activation": "geglu", "residual": False},
        # a transformer block of the 1280-wide level (60 of the UNet's 70), one image
        dict({"name": "block_1280_e4m3", "kind": "block", "channels": 1280, "dtype": "e4m3", "scales": "channel", "group": 0},
             **image(1)),
        # the same level in INT8 for a portrait image: a row count that is no multiple of the tile
        dict({"name": "block_1280_int8_portrait", "kind": "block", "channels": 1280, "dtype": "int8", "scales": "channel",
              "group": 256}, **image(1, 1216, 832)),
        # the 640-wide level in INT8, one image
        dict({"name": "block_640_int8", "kind": "block", "channels": 640, "dtype": "int8", "scales": "channel", "group": 256},
             **image(1)),
        # the 640-wide level in FP8 for a batch of eight images: the largest activations of the loop
        dict({"name": "block_640_e4m3_batch", "kind": "block", "channels": 640, "dtype": "e4m3", "scales": "channel",
              "group": 0}, **image(8)),
        # all 140 cross-attention K / V projections of one prompt pair: weights streamed once
        {"name": "cross_kv_int8", "kind": "cross_kv", "images": 1, "dtype": "int8", "scales": "channel", "group": 256},
        # every projection of a step as one grouped plan
        dict({"name": "projections_e5m2", "kind": "projections", "dtype": "e5m2", "scales": "channel", "group": 0}, **image(1)),
        # packing a block's weights when a checkpoint is loaded
        {"name": "load_block_1280_int8", "kind": "load", "channels": 1280, "source": "f16", "dtype": "int8",
         "scales": "channel", "group": 256},
        # one denoising step of the whole UNet, one image
        dict({"name": "denoise_e4m3", "kind": "denoise", "dtype": "e4m3", "scales": "channel", "group": 0}, **image(1)),
    ]


def _precision(rng, weights_only=False):
    dtype = rng.choice(["int8", "int8", "e4m3", "e4m3", "e5m2"] + ([] if weights_only else ["f16"]))
    if dtype == "int8":
        return {"dtype": dtype, "scales": "channel", "group": rng.choice([256, 256, 256, 64, 0])}
    if dtype == "f16":
        return {"dtype": dtype, "scales": "none", "group": 0}
    return {"dtype": dtype, "scales": rng.choice(["channel", "channel", "tensor"]), "group": 0}


def _size(rng, largest):
    return {"height": 64 * rng.randint(8, largest // 64), "width": 64 * rng.randint(8, largest // 64)}


def _log_uniform(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choices(["linear", "block", "cross_kv", "projections", "load", "denoise"], [40, 28, 9, 6, 10, 7])[0]
    if kind == "linear":
        # (n, k, activation, residual, most rows) of the path's projections and the text encoders' fully connected layers
        role = rng.choice(["square", "out", "geglu", "down", "context", "time", "label", "text_up", "text_down"])
        c = rng.choice([640, 1280])
        most = {640: 65536, 1280: 16384}[c]
        e, act = rng.choice([(768, "quick_gelu"), (1280, "gelu")])
        n, k, activation, residual, rows = {
            "square": (c, c, "none", False, most), "out": (c, c, "none", True, most), "geglu": (8 * c, c, "geglu", False, most),
            "down": (c, 4 * c, "none", True, most), "context": (c, CROSS_DIM, "none", False, 1232),
            "time": (1280, 320, "silu", False, 16), "label": (1280, 2816, "silu", False, 16),
            "text_up": (4 * e, e, act, False, 1232), "text_down": (e, 4 * e, "none", False, 1232)}[role]
        return dict({"kind": kind, "m": _log_uniform(rng, 1, rows), "n": n, "k": k, "activation": activation,
                     "residual": residual}, **_precision(rng))
    if kind == "block":
        return dict({"kind": kind, "channels": rng.choice([640, 1280]), "images": _log_uniform(rng, 1, 8)},
                    **_size(rng, 1024), **_precision(rng))
    if kind == "cross_kv":
        return dict({"kind": kind, "images": rng.randint(1, 16)}, **_precision(rng))
    if kind == "load":
        return dict({"kind": kind, "channels": rng.choice([640, 1280]), "source": rng.choice(["f16", "f32"])},
                    **_precision(rng, weights_only=True))
    return dict({"kind": kind, "images": 1}, **_size(rng, 1024), **_precision(rng))


# ---- what a program holds before the call -----------------------------------------------------------
@functools.lru_cache(maxsize=None)
def operator():
    """The one context and operator object a program keeps for its GPU."""
    return pkg.Ops(pkg.Context(torch.cuda.current_device(), workspace_bytes=3 << 30))


class Source:
    """Seeded tensors on the GPU."""

    def __init__(self, seed):
        self.generator = torch.Generator(device="cuda")
        self.generator.manual_seed(seed & 0x7FFFFFFF)

    def normal(self, *shape, scale=1.0, shift=0.0, dtype=torch.float16):
        x = torch.randn(shape, generator=self.generator, device="cuda", dtype=torch.float32)
        return x.mul_(scale).add_(shift).to(dtype)

    def activations(self, *shape):
        """N(0, 1) with one channel in a hundred at 20 times the size, like the hidden states of the model."""
        x = torch.randn(shape, generator=self.generator, device="cuda", dtype=torch.float32)
        loud = torch.randperm(shape[-1], generator=self.generator, device="cuda")[: max(1, shape[-1] // 100)]
        x[..., loud] *= 20.0
        return x.half()

    def matrix(self, n, k, dtype=torch.float16):
        return self.normal(n, k, scale=k ** -0.5, dtype=dtype)


def pack(case, source):
    ops = operator()
    if case["dtype"] == "f16":
        return ops.fp16_weight(source)
    if case["dtype"] == "int8":
        return ops.upload_or_quantize_int8_weight(source, None, pkg.INT8WeightLoadOptions(
            enable_convrot=case["group"] != 0, convrot_group_size=case["group"]))
    fmt = {"e4m3": pkg.ScalarType.Float8E4M3, "e5m2": pkg.ScalarType.Float8E5M2}[case["dtype"]]
    mode = {"channel": pkg.FP8ScaleMode.PerOutputChannel, "tensor": pkg.FP8ScaleMode.TensorWide}[case["scales"]]
    return ops.upload_fp8_weight(source, pkg.FP8WeightLoadOptions(format=fmt, scale_mode=mode))


def block_weights(c):
    """(name, n, k, bias) of a transformer block's projections."""
    return [("to_q", c, c, False), ("to_k", c, c, False), ("to_v", c, c, False), ("to_out", c, c, True),
            ("cross_q", c, c, False), ("cross_k", c, CROSS_DIM, False), ("cross_v", c, CROSS_DIM, False),
            ("cross_out", c, c, True), ("up", 8 * c, c, True), ("down", c, 4 * c, True)]


def cross_projections(images):
    return [p for p in shapes.unet_projections(2 * images) if p.k == CROSS_DIM]


def grouped(source, case, projections):
    """A plan over the projections, its outputs laid out in one buffer."""
    inputs, places, total = {}, [], 0
    for p in projections:
        if p.input_key not in inputs:
            inputs[p.input_key] = source.activations(p.m, p.k)
        n_out = p.n // 2 if p.activation == pkg.ACT_GEGLU else p.n
        places.append((total, p.m, n_out))
        total += -(-p.m * n_out // 128) * 128
    outputs = torch.zeros(total, dtype=torch.float16, device="cuda")
    calls = []
    for p, (at, m, n_out) in zip(projections, places):
        bias = source.normal(p.n, scale=0.1) if p.bias else None
        calls.append(pkg.LinearCall(inputs[p.input_key], pack(case, source.matrix(p.n, p.k)), bias, p.activation,
                                    outputs[at:at + m * n_out].view(m, n_out)))
    return {"plan": operator().plan(calls), "outputs": outputs}


def prepare(case, seed):
    kind, source = case["kind"], Source(seed)
    state = {"kind": kind, "case": case, "ops": operator()}
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        state["x"] = source.activations(m, k)
        state["weight"] = pack(case, source.matrix(n, k))
        state["bias"] = source.normal(n, scale=0.1)
        state["residual"] = source.activations(m, n) if case["residual"] else None
        state["activation"] = ACTIVATIONS[case["activation"]]
    elif kind == "block":
        c = case["channels"]
        m = tokens(case, c)
        state["hidden"] = source.activations(m, c)
        state["attention"] = [source.normal(m, c), source.normal(m, c)]
        state["norms"] = [(source.normal(c, scale=0.05, shift=1.0), source.normal(c, scale=0.02)) for _ in range(3)]
        for name, n, k, bias in block_weights(c):
            if k != CROSS_DIM:                      # the context's K and V are projected once per generation
                state[name] = pack(case, source.matrix(n, k))
                state[name + ".bias"] = source.normal(n, scale=0.02) if bias else None
        # FP8: the word through which the feed-forward's first projection hands its output's maximum on
        state["amax"] = torch.zeros(1, dtype=torch.int32, device="cuda") if case["dtype"] in ("e4m3", "e5m2") else None
    elif kind == "cross_kv":
        state.update(grouped(source, case, cross_projections(case["images"])))
    elif kind == "projections":
        state.update(grouped(source, case, shapes.unet_projections(2 * case["images"], case["height"], case["width"])))
    elif kind == "load":
        dtype = {"f16": torch.float16, "f32": torch.float32}[case["source"]]
        state["sources"] = [source.matrix(n, k, dtype) for _, n, k, _ in block_weights(case["channels"])]
    else:
        torch.backends.cudnn.benchmark = True       # the convolutions around the path: algorithms picked at warm-up
        images, config = case["images"], pkg.unet_harness.BASE_1_0
        unet = DenoiseUNet(state["ops"], case, seed)
        loop = pkg.EulerDenoiser(unet, images, case["height"], case["width"], steps=20)
        ids = torch.tensor([[case["height"], case["width"], 0, 0, case["height"], case["width"]]], dtype=torch.float16)
        loop.set_conditioning(source.normal(2 * images, CONTEXT_TOKENS, config.cross_attention_dim),
                              source.normal(2 * images, config.pooled_dim), ids.repeat(2 * images, 1).cuda())
        state["noise"] = source.normal(*loop.latents.shape, dtype=torch.float32)
        state["loop"] = loop
        loop.set_latents(state["noise"])
        loop.step()                                 # records the step's graph
    return state


class DenoiseUNet(pkg.UNetHarness):
    """The UNet with the case's packing of its projection weights."""

    def __init__(self, ops, case, seed):
        self.case = case
        super().__init__(ops, precision=case["dtype"], seed=seed)

    def _pack(self, values):
        return pack(self.case, values.to(torch.float16))


# ---- one pass -----------------------------------------------------------------------------------------
def run_block(s):
    ops, hidden = s["ops"], s["hidden"]

    def norm(x, index, consumer):
        gamma, beta = s["norms"][index]
        if s["case"]["dtype"] == "f16":
            return {"input": ops.layer_norm(x, gamma, beta)}
        xq, scales = ops.layer_norm_quantized(x, gamma, beta, s[consumer])
        return {"input": None, "xq": xq, "xq_scales": scales}

    first = norm(hidden, 0, "to_q")
    qkv = ops.linear_grouped([pkg.LinearCall(first["input"], s[name], xq=first.get("xq"), xq_scales=first.get("xq_scales"))
                              for name in ("to_q", "to_k", "to_v")])
    # the caller's tensor is kept; from here on the hidden state is updated in place
    hidden = ops.linear(s["attention"][0], s["to_out"], s["to_out.bias"], residual=hidden)
    query = ops.linear(weight=s["cross_q"], **norm(hidden, 1, "cross_q"))
    hidden = ops.linear(s["attention"][1], s["cross_out"], s["cross_out.bias"], residual=hidden, out=hidden)
    wide = ops.linear_activation(weight=s["up"], bias=s["up.bias"], activation=pkg.ACT_GEGLU, y_amax=s["amax"],
                                 **norm(hidden, 2, "up"))
    hidden = ops.linear(wide, s["down"], s["down.bias"], residual=hidden, out=hidden, x_amax=s["amax"])
    return qkv + [query, hidden]


def run(state):
    kind, ops = state["kind"], state["ops"]
    if kind == "linear":
        if state["activation"] == pkg.ACT_NONE:
            return ops.linear(state["x"], state["weight"], state["bias"], residual=state["residual"])
        return ops.linear_activation(state["x"], state["weight"], state["bias"], state["activation"])
    if kind == "block":
        return run_block(state)
    if kind == "load":
        packed = [pack(state["case"], source) for source in state["sources"]]
        return [t for w in packed for t in (w.data, w.scales)]
    if kind == "denoise":
        state["loop"].set_latents(state["noise"])
        state["loop"].step()
        return state["loop"].latents
    state["plan"].run()
    return state["outputs"]


# ---- what a pass cannot do without ----------------------------------------------------------------------
def _weight_bytes(case, n, k):
    if case["dtype"] == "f16":
        return 2 * n * k
    return n * k + 4 * (n if case["scales"] == "channel" else 1)


def work(case):
    kind = case["kind"]
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        n_out = n // 2 if case["activation"] == "geglu" else n
        return {"bytes": 2 * m * k + _weight_bytes(case, n, k) + 2 * n + 2 * m * n_out * (2 if case["residual"] else 1),
                "flops": 2 * m * n * k}
    if kind == "block":
        c = case["channels"]
        m = tokens(case, c)
        weights = [(n, k) for _, n, k, _ in block_weights(c) if k != CROSS_DIM]
        # in: hidden, two attention results; out: q, k, v, the cross-attention query, hidden
        return {"bytes": sum(_weight_bytes(case, n, k) for n, k in weights) + 2 * m * c * 8,
                "flops": sum(2 * m * n * k for n, k in weights)}
    if kind == "load":
        element = {"f16": 2, "f32": 4}[case["source"]]
        return {"bytes": sum(element * n * k + _weight_bytes(case, n, k) for _, n, k, _ in block_weights(case["channels"])),
                "flops": 0}
    if kind == "cross_kv":
        projections = cross_projections(case["images"])
    else:
        projections = shapes.unet_projections(2 * case["images"], case["height"], case["width"])
    flops = sum(2 * p.m * p.n * p.k for p in projections)
    weights = sum(_weight_bytes(case, p.n, p.k) for p in projections)
    if kind == "denoise":
        # the projections and 3x3 / 1x1 convolutions of a step; attention scores are left out
        at, convolutions, weight_values = _convolution_sizes(case)
        return {"bytes": weights + 2 * weight_values + 8 * 4 * case["images"] * at, "flops": flops + convolutions}
    inputs = {p.input_key: p.m * p.k for p in projections}
    outputs = sum(p.m * (p.n // 2 if p.activation == pkg.ACT_GEGLU else p.n) for p in projections)
    return {"bytes": weights + 2 * sum(inputs.values()) + 2 * outputs, "flops": flops}


def _convolution_sizes(case):
    """(latent pixels, operations, weight values) of the UNet's convolutions; each at the resolution of its block."""
    pixels = (case["height"] // 8) * (case["width"] // 8)
    operations, values = 0, 0
    for name, shape in pkg.unet_harness.unet_parameter_shapes().items():
        if len(shape) != 4:
            continue
        level = 0
        if name.startswith("down_blocks."):
            level = int(name.split(".")[1]) + (1 if "downsamplers" in name else 0)
        elif name.startswith("mid_block."):
            level = 2
        elif name.startswith("up_blocks."):
            level = 2 - int(name.split(".")[1]) - (1 if "upsamplers" in name else 0)
        count = math.prod(shape)
        values += count
        operations += 2 * count * 2 * case["images"] * (pixels >> (2 * level))
    return pixels, operations, values


def tolerance(case):
    kind, dtype = case["kind"], case["dtype"]
    if kind == "load":
        return "exact"
    # FP16 results of FP32 or integer sums: half an ulp is 2^-11, and results near a tie may round either way
    rel = {"int8": 1e-3, "f16": 1e-3, "e4m3": 2e-3, "e5m2": 2e-3}[dtype]
    if kind == "block":
        # another order of a norm's sums moves its FP16 results at ties, and with them the quantised values; a tensor-wide
        # FP8 scale that moves by one FP16 ulp moves one value in a hundred by a step of 2^-3 (E4M3) or 2^-2 (E5M2)
        rel = {"int8": 5e-3, "f16": 2e-3, "e4m3": 1e-2, "e5m2": 2e-2}[dtype]
    if kind == "denoise":
        rel = 1e-2          # the same through the whole network; the step adds its prediction to the latents
    return {"rel": rel}
