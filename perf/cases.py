"""Workloads that a user of this package runs, with their inputs, the work they cannot do without and the
tolerance of their results.

Sizes are those of the texture UNet's linear layers (2 x 6 views at 64 x 64, 32 x 32 and 16 x 16 tokens,
channels 320 / 640 / 1280), of the image encoder's (257 tokens, 1536 / 6144 wide) and ragged ones around
them.  A case is one call through the public modules: ``Int8Linear`` (dense and 2:4 sparse, plain, GELU and
GEGLU epilogues), ``Int8LayerNorm`` + ``Int8Linear``, ``GroupNormNHWC``, the conversion of an ``nn.Linear``,
and a whole UNet forward, replayed from a CUDA graph or eager.
"""
import functools
import importlib
import math

import torch
import torch.nn as nn

PKG = "hunyuan3d-tools_b200"
DEV = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _mod(name):
    return importlib.import_module(PKG + "." + name)


def _linear(name, batch, rows, k, n, mode="dense", epilogue="linear", bias=True, dtype="bf16"):
    return {"name": name, "kind": "linear", "mode": mode, "batch": batch, "rows": rows, "k": k, "n": n,
            "epilogue": epilogue, "bias": bias, "dtype": dtype}


def listed():
    return [
        # The smallest layer of a denoise step: the time-embedding projection of a ResNet block, one row
        # per sample.  22 of them run in every step.
        _linear("time_proj_12x1280x640", 12, 1, 1280, 640),
        # Cross-attention keys and values stacked: 12 samples x 77 text tokens, no bias.
        _linear("cross_kv_924x1024x2560", 12, 77, 1024, 2560, bias=False),
        # Image encoder's second MLP layer: one image of 257 tokens, few rows and a deep K.
        _linear("encoder_fc2_257x6144x1536", 1, 257, 6144, 1536, dtype="fp16"),
        # proj_in / proj_out / attention output at the highest resolution: many rows, everything else short.
        _linear("attn_out_49152x320x320", 12, 4096, 320, 320),
        # Feed-forward up-projection with its GEGLU gate at the highest resolution.
        _linear("ffn_up_geglu_49152x320x2560", 12, 4096, 320, 2560, epilogue="geglu"),
        # Feed-forward down-projection at the middle resolution.
        _linear("ffn_down_12288x2560x640", 12, 1024, 2560, 640),
        # LayerNorm that hands int8 codes to the stacked q / k / v projection.
        {"name": "ln_qkv_12288x640x1920", "kind": "ln_linear", "batch": 12, "rows": 1024, "k": 640, "n": 1920,
         "bias": False, "dtype": "bf16"},
        # 2:4-sparse feed-forward up-projection with its gate at the lowest resolution, the layer the
        # mixed mode assigns to the sparse kernel.
        _linear("sparse_up_geglu_3072x1280x10240", 12, 256, 1280, 10240, mode="sparse", epilogue="geglu"),
        # 2:4-sparse down-projection on a ragged token count (5 views of a non-square crop), fp16 with GELU.
        _linear("sparse_gelu_2915x5120x1296", 5, 583, 5120, 1296, mode="sparse", epilogue="gelu", dtype="fp16"),
        # GroupNorm + SiLU with the time-embedding term of a ResNet block, channels last.
        {"name": "groupnorm_12x320x64x64", "kind": "groupnorm", "batch": 12, "c": 320, "h": 64, "w": 64,
         "silu": True, "add": True, "dtype": "bf16"},
        # Loading a model: one nn.Linear quantised, pruned 2:4, compressed and packed on the GPU.
        {"name": "convert_sparse_10240x1280", "kind": "convert", "mode": "sparse", "k": 1280, "n": 10240,
         "bias": True, "dtype": "bf16"},
        # A denoise step: the full UNet on [uncond | cond] x 6 views of 64 x 64 latents, mixed dense /
        # sparse INT8 layers, replayed from its CUDA graph as the mesh driver does.
        {"name": "unet_step_6view_64", "kind": "unet", "views": 6, "size": 64, "width": 320, "quant": "mixed",
         "graph": True},
    ]


MAX_MNK = 49152 * 320 * 2560
MAX_ELEMENTS = 49152 * (320 + 2560)


def _log(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi, max(lo, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choices(["linear", "sparse", "ln_linear", "groupnorm", "convert", "unet"],
                       weights=[36, 16, 14, 12, 10, 12])[0]
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    bias = rng.random() < 0.7
    if kind == "groupnorm":
        while True:
            case = {"kind": kind, "batch": rng.randint(1, 12), "c": _log(rng, 64, 2560, 32), "h": _log(rng, 6, 96),
                    "w": _log(rng, 6, 96), "silu": rng.random() < 0.7, "add": rng.random() < 0.4, "dtype": dtype}
            if case["batch"] * case["c"] * case["h"] * case["w"] <= 12 * 960 * 64 * 64:
                return case
    if kind == "convert":
        return {"kind": kind, "mode": rng.choice(["sparse", "sparse", "dense"]), "k": _log(rng, 128, 6144, 64),
                "n": _log(rng, 128, 10240, 16), "bias": bias, "dtype": rng.choice(["bf16", "fp16", "fp32"])}
    if kind == "unet":
        return {"kind": kind, "views": rng.randint(1, 6), "size": 8 * rng.randint(2, 8), "width": 64 * rng.randint(2, 5),
                "quant": rng.choice(["mixed", "dense"]), "graph": rng.random() < 0.6}
    while True:
        batch = rng.choice([1, 1, 2, 5, 6, 12])
        rows = _log(rng, 1, 8192)
        k = _log(rng, 640 if kind == "sparse" else 128, 2048 if kind == "ln_linear" else 6144, 64)
        n = _log(rng, 128, 10240, 32)
        if rng.random() < 0.3:
            n += 16
        m = batch * rows
        if m <= 49152 and m * k * n <= MAX_MNK and m * (k + n) <= MAX_ELEMENTS:
            break
    if kind == "ln_linear":
        return {"kind": kind, "batch": batch, "rows": rows, "k": k, "n": n, "bias": bias, "dtype": dtype}
    epilogue = rng.choice(["linear", "linear", "gelu", "geglu"])
    if epilogue == "geglu":
        n -= n % 32
    return {"kind": "linear", "mode": "sparse" if kind == "sparse" else "dense", "batch": batch, "rows": rows, "k": k,
            "n": n, "epilogue": epilogue, "bias": bias, "dtype": dtype}


# ---------------------------------------------------------------------------------------
# what a program has in hand before the call
# ---------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _activation(g, shape, dtype):
    """N(0,1) with 0.1 % of the entries at +-20, as the linear layers' inputs."""
    x = torch.randn(shape, generator=g, device=DEV)
    u = torch.rand(shape, generator=g, device=DEV)
    x = torch.where(u < 0.0005, 20.0, torch.where(u > 0.9995, -20.0, x))
    return x.to(dtype)


def _nn_linear(g, k, n, bias, dtype):
    lin = nn.Linear(k, n, bias=bias, device=DEV, dtype=dtype)
    lin.weight.data.copy_(torch.randn(n, k, generator=g, device=DEV) * 0.02)
    if bias:
        lin.bias.data.copy_(torch.randn(n, generator=g, device=DEV) * 0.01)
    return lin


def _tokens(case):
    return (case["batch"], case["k"]) if case["rows"] == 1 else (case["batch"], case["rows"], case["k"])


def _unet_config(case):
    w = case["width"]
    return {"block_out_channels": (w, 2 * w, 4 * w, 4 * w), "attention_heads": (w // 64, w // 32, w // 16, w // 16),
            "num_views": case["views"]}


def prepare(case, seed):
    qu = _mod("quantize_utils")
    g = _gen(seed)
    kind = case["kind"]
    if kind == "unet":
        mm = _mod("multimesh")
        unet, _ = mm.build_texture_unet(DEV, torch.bfloat16, case["quant"], seed=seed, init_on_device=True,
                                        **_unet_config(case))
        batch, size = 2 * case["views"], case["size"]
        lat = torch.randn(case["views"], 4, size, size, generator=g, device=DEV).bfloat16()
        cond = torch.randn(case["views"], 77, 1024, generator=g, device=DEV).bfloat16()
        step = mm.GraphedStep(unet, batch, size, 77, 1024, torch.bfloat16, DEV) if case["graph"] else unet
        # the captured step reads the model's weights: the program keeps both
        return {"kind": kind, "unet": unet, "step": step, "x": torch.cat([lat, lat]),
                "t": torch.full((batch,), 100 + seed % 800, device=DEV),
                "ctx": torch.cat([torch.zeros_like(cond), cond])}
    dtype = DTYPES[case["dtype"]]
    if kind == "groupnorm":
        norm = _mod("unet").GroupNormNHWC(32, case["c"], eps=1e-5, silu=case["silu"]).to(DEV).to(dtype)
        norm.weight.data.copy_(1.0 + 0.1 * torch.randn(case["c"], generator=g, device=DEV))
        norm.bias.data.copy_(0.1 * torch.randn(case["c"], generator=g, device=DEV))
        norm.requires_grad_(False).fused = True
        x = torch.randn(case["batch"], case["c"], case["h"], case["w"], generator=g, device=DEV).to(dtype)
        add = torch.randn(case["batch"], case["c"], generator=g, device=DEV).to(dtype) if case["add"] else None
        return {"kind": kind, "norm": norm, "x": x.contiguous(memory_format=torch.channels_last), "add": add}
    lin = _nn_linear(g, case["k"], case["n"], case["bias"], dtype)
    if kind == "convert":
        make = qu.Int8Linear.from_linear_sparse if case["mode"] == "sparse" else qu.Int8Linear.from_linear
        return {"kind": kind, "make": make, "lin": lin}
    x = _activation(g, _tokens(case), dtype)
    if kind == "ln_linear":
        ln = nn.LayerNorm(case["k"], device=DEV, dtype=dtype)
        ln.weight.data.copy_(1.0 + 0.1 * torch.randn(case["k"], generator=g, device=DEV))
        ln.bias.data.copy_(0.1 * torch.randn(case["k"], generator=g, device=DEV))
        return {"kind": kind, "norm": qu.Int8LayerNorm(ln), "layer": qu.Int8Linear.from_linear(lin), "x": x}
    make = qu.Int8Linear.from_linear_sparse if case["mode"] == "sparse" else qu.Int8Linear.from_linear
    layer = make(lin)
    if case["epilogue"] == "geglu":
        layer.interleave_geglu_rows()
    else:
        layer.epilogue = case["epilogue"]
    return {"kind": kind, "layer": layer, "x": x}


@torch.no_grad()
def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["layer"](state["x"])
    if kind == "ln_linear":
        return state["layer"](state["norm"](state["x"]))
    if kind == "groupnorm":
        return state["norm"](state["x"], state["add"])
    if kind == "convert":
        layer = state["make"](state["lin"])
        return [layer.weight_int8_nk, layer.weight_sparse_comp, layer.weight_sparse_meta, layer.weight_scale, layer.bias]
    return state["step"](state["x"], state["t"], state["ctx"])


# ---------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _unet_work(views, size, width):
    """Operations of one forward counted by torch on the meta device; bytes: every weight once (linear layers
    one byte, the rest two) and the step's inputs and output."""
    from torch.utils.flop_counter import FlopCounterMode
    with torch.device("meta"):
        net = _mod("unet").UNetSD21MV(**_unet_config({"views": views, "width": width}))
        b = 2 * views
        args = (torch.empty(b, 4, size, size), torch.empty(b, dtype=torch.long), torch.empty(b, 77, 1024))
        with FlopCounterMode(display=False) as counter, torch.no_grad():
            net(*args)
    linear = sum(m.weight.numel() for m in net.modules() if isinstance(m, nn.Linear))
    total = sum(p.numel() for p in net.parameters())
    io = 2 * (2 * args[0].numel() + args[2].numel())
    return {"bytes": linear + 2 * (total - linear) + io, "flops": counter.get_total_flops()}


def work(case):
    kind = case["kind"]
    if kind == "unet":
        return _unet_work(case["views"], case["size"], case["width"])
    if kind == "groupnorm":
        n = case["batch"] * case["c"] * case["h"] * case["w"]
        return {"bytes": 4 * n + 4 * case["c"], "flops": 8 * n}
    k, n = case["k"], case["n"]
    if kind == "convert":
        src = 4 if case["dtype"] == "fp32" else 2
        return {"bytes": n * k * (src + (0.625 if case["mode"] == "sparse" else 1)) + 8 * n, "flops": 3 * n * k}
    m = case["batch"] * case["rows"]
    sparse = case.get("mode") == "sparse"
    n_out = n // 2 if case.get("epilogue") == "geglu" else n
    return {"bytes": 2 * m * k + 2 * m * n_out + n * k * (0.625 if sparse else 1) + 4 * n,
            "flops": m * n * k * (1 if sparse else 2)}


def tolerance(case):
    kind = case["kind"]
    if kind == "unet":
        return {"rel": 2e-2}                  # bf16 throughout; a changed rounding moves int8 codes downstream
    if kind == "convert":
        return {"rel": 4e-3}                  # codes and metadata the same; scales are 16-bit values
    bf16 = case["dtype"] == "bf16"
    if kind == "ln_linear":
        return {"rel": 1e-2 if bf16 else 4e-3}   # the normalised row is rounded, then quantised to 8 bits
    if kind == "groupnorm":
        return {"rel": 6e-3 if bf16 else 1e-3}   # up to three roundings to the 16-bit type
    return {"rel": 4e-3 if bf16 else 1e-3}    # exact int32 sums, one rounding to the 16-bit type
