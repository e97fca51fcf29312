"""The work that this package is timed on: DP layers called as a training program calls them.

A case is one pass through the public entry points -- a DP layer's forward and backward, one backward
through the operator functions, or the forward and backward of a wrapped transformer stack -- and the pass
returns everything it computes: outputs, input gradients and parameter gradients.

Kinds of case:
  linear / conv1d   `DPLinear` / `DPConv1D`, forward and backward.  `t` = 0 is a 2-D input of `b` samples.
  linear_bwd        the backward alone through `flashdp4review_b200.core` (weight gradient with norms and
                    factors, input gradient).
  layernorm         `DPLayerNorm`, forward and backward.
  stack             GPT-2 style blocks put through `wrap_with_flashdp_layers`, bf16 autocast over fp32
                    parameters, forward and backward.
"""
import math

import torch
import torch.nn as nn
import torch.nn.functional as F

from flashdp4review_b200 import DPConv1D, DPLayerNorm, DPLinear, manual_seed, wrap_with_flashdp_layers
from flashdp4review_b200 import core
from flashdp4review_b200.layers import Conv1D

_DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16}
_NOISE_KEY = 20240229     # one fixed noise key: two runs of a case draw the same noise


def _linear(name, b, t, n_in, n_out, dtype, *, kind="linear", bias=True, autocast=False, g_scale=1e-3, noise=1.0):
    return {"name": name, "kind": kind, "b": b, "t": t, "n_in": n_in, "n_out": n_out, "dtype": dtype, "bias": bias,
            "autocast": autocast, "g_scale": g_scale, "noise": noise}


def _layernorm(name, b, t, d, dtype, noise=1.0):
    return {"name": name, "kind": "layernorm", "b": b, "t": t, "d": d, "dtype": dtype, "g_scale": 1e-3, "noise": noise}


def listed():
    return [
        # the repository's small single-layer configuration in the default dtype: launches and host time
        _linear("linear_fp32_b4_t128_768x768", 4, 128, 768, 768, "fp32", g_scale=1e-2),
        # a classifier head over pooled features, one row per sample
        _linear("linear_fp32_b1024_1024x1000", 1024, 0, 1024, 1000, "fp32", g_scale=1e-2, noise=0.0),
        # an MLP layer of an image transformer (196 patches and a class token) in the default dtype
        _linear("linear_fp32_b16_t197_768x3072", 16, 197, 768, 3072, "fp32", g_scale=1e-2, noise=0.0),
        # GPT-2-medium's attention projection in the default dtype, micro-batch 8
        _linear("conv1d_fp32_b8_t1024_1024x3072", 8, 1024, 1024, 3072, "fp32", kind="conv1d"),
        # short padded sentences, fine-tuned under autocast
        _linear("linear_amp_b32_t77_768x768", 32, 77, 768, 768, "bf16", autocast=True, noise=0.0),
        # sequences that no tile size divides, fp16
        _linear("linear_fp16_b12_t500_1024x4096", 12, 500, 1024, 4096, "fp16", noise=0.0),
        # the repository's GPT-2 attention projection configuration
        _linear("conv1d_bf16_b16_t1024_1024x3072", 16, 1024, 1024, 3072, "bf16", kind="conv1d"),
        # the LayerNorm of the same configuration
        _layernorm("layernorm_bf16_b16_t1024_d1024", 16, 1024, 1024, "bf16"),
        # a small LayerNorm in the default dtype
        _layernorm("layernorm_fp32_b6_t197_d768", 6, 197, 768, "fp32", noise=0.0),
        # two GPT-2-medium blocks, micro-batch 8: every wrapped layer kind in the order of a training step
        {"name": "stack_amp_2x1024_b8_t1024", "kind": "stack", "blocks": 2, "width": 1024, "heads": 16, "b": 8, "t": 1024,
         "g_scale": 1e-3, "noise": 1.0},
        # the headline configuration: backward of a 4096 x 4096 layer
        _linear("linear_bwd_bf16_b32_t1024_4096x4096", 32, 1024, 4096, 4096, "bf16", kind="linear_bwd", bias=False),
        # the up-projection of the Llama-2-7B-shaped decoder, micro-batch 4
        _linear("linear_bf16_b4_t2048_4096x11008", 4, 2048, 4096, 11008, "bf16", bias=False),
    ]


# ---- drawn cases -------------------------------------------------------------------------------------
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, lo, hi):
    """A layer width: mostly multiples of 64, some of 8 only, now and then any number."""
    n = _log_int(rng, lo, hi)
    step = rng.choice([64, 64, 64, 8, 8, 1])
    return max(lo, n // step * step)


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "conv1d", "conv1d", "linear_bwd", "layernorm", "layernorm", "stack"])
    noise = rng.choice([0.0, 1.0])
    if kind == "stack":
        heads = rng.choice([4, 8, 12, 16])
        return {"kind": kind, "blocks": rng.choice([1, 2]), "width": 64 * heads, "heads": heads, "b": rng.randint(2, 8),
                "t": _log_int(rng, 32, 1024), "g_scale": 1e-3, "noise": noise}
    dtype = rng.choice(["fp32", "fp32", "bf16", "bf16", "fp16"])
    if kind == "layernorm":
        d = _width(rng, 64, 8192)
        b = rng.randint(1, 32)
        t = min(_log_int(rng, 16, 4096), max(1, 24_000_000 // (b * d)))
        c = _layernorm(None, b, t, d, dtype, noise)
    else:
        autocast = dtype != "fp32" and kind != "linear_bwd" and rng.random() < 0.3
        n_in, n_out = _width(rng, 64, 8192), _width(rng, 64, 8192)
        if kind == "linear" and rng.random() < 0.2:
            b, t = _log_int(rng, 16, 4096), 0
        else:
            b, t = _log_int(rng, 1, 64), rng.choice([_log_int(rng, 2, 4096), 64 * _log_int(rng, 1, 64)])
        # fp32 passes are held to a tenth of the 16-bit ones' work
        most = (1.5e11 if dtype == "fp32" else 1.5e12) / (6.0 * n_in * n_out)
        if t:
            t = max(2, min(t, int(most / b), 65536 // b))
        else:
            b = max(16, min(b, int(most)))
        c = _linear(None, b, t, n_in, n_out, dtype, kind=kind, bias=kind != "linear_bwd" and rng.random() < 0.7, autocast=autocast,
                    g_scale=rng.choice([1e-2, 1e-3]), noise=noise)
        if kind == "conv1d":
            c["bias"] = True
    del c["name"]
    return c


# ---- one pass ----------------------------------------------------------------------------------------
class _Block(nn.Module):
    """A GPT-2 block: pre-norm attention and MLP, Conv1D projections."""

    def __init__(self, width, heads):
        super().__init__()
        self.heads = heads
        self.ln_1, self.ln_2 = nn.LayerNorm(width), nn.LayerNorm(width)
        self.c_attn, self.c_proj = Conv1D(3 * width, width), Conv1D(width, width)
        self.c_fc, self.c_out = Conv1D(4 * width, width), Conv1D(width, 4 * width)

    def forward(self, x):
        B, T, D = x.shape
        q, k, v = (p.view(B, T, self.heads, -1).transpose(1, 2) for p in self.c_attn(self.ln_1(x)).split(D, dim=2))
        a = F.scaled_dot_product_attention(q, k, v, is_causal=True)
        x = x + self.c_proj(a.transpose(1, 2).reshape(B, T, D))
        return x + self.c_out(F.gelu(self.c_fc(self.ln_2(x)), approximate="tanh"))


def _pin_noise(model):
    """Fixed noise streams: the ids that select them otherwise count every layer the process has built."""
    n = 0
    for m in model.modules():
        if getattr(m, "dp", False):
            m._dp_param_ids = [n + 1, n + 2]
            n += 2


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, scale=1.0, dtype=torch.float32):
        return (torch.randn(*shape, device="cuda", generator=gen) * scale).to(dtype)

    manual_seed(_NOISE_KEY)
    s = {"case": case}
    kind = case["kind"]
    hyper = dict(C=1.0, clamp_value=1.0, noise_multiplier=case["noise"])
    if kind == "stack":
        model = nn.Sequential(*[_Block(case["width"], case["heads"]) for _ in range(case["blocks"])]).cuda()
        with torch.no_grad():
            for m in model.modules():
                if isinstance(m, Conv1D):
                    m.weight.normal_(0.0, 0.02, generator=gen)
                    m.bias.zero_()
        s["layer"] = wrap_with_flashdp_layers(model, target_modules=[Conv1D, nn.LayerNorm], feedback=False, **hyper)
        shape, width, dtype, autocast = (case["b"], case["t"]), case["width"], torch.float32, True
        n_out = width
    elif kind == "layernorm":
        dtype, autocast, width = _DTYPES[case["dtype"]], False, case["d"]
        s["layer"] = DPLayerNorm(width, device="cuda", dtype=dtype, use_fused=False, **hyper)
        with torch.no_grad():
            s["layer"].weight.copy_(1.0 + normal(width, scale=0.1))
            s["layer"].bias.copy_(normal(width, scale=0.1))
        shape, n_out = (case["b"], case["t"]), width
    else:
        dtype, autocast, width, n_out = _DTYPES[case["dtype"]], case["autocast"], case["n_in"], case["n_out"]
        shape = (case["b"], case["t"]) if case["t"] else (case["b"],)
        pdtype = torch.float32 if autocast else dtype
        if kind == "linear_bwd":
            s["weight"] = normal(n_out, width, scale=0.02, dtype=dtype)
        else:
            if kind == "conv1d":
                layer = DPConv1D(n_out, width, **hyper).to(device="cuda", dtype=pdtype)
            else:
                layer = DPLinear(width, n_out, bias=True if case["bias"] else None, device="cuda", dtype=pdtype, **hyper)
            with torch.no_grad():
                layer.weight.copy_(normal(*layer.weight.shape, scale=0.02))
                if layer.bias is not None:
                    layer.bias.copy_(normal(n_out, scale=0.02))
            s["layer"] = layer
    if "layer" in s:
        _pin_noise(s["layer"])
    s["autocast"] = (_DTYPES[case["dtype"]] if kind != "stack" else torch.bfloat16) if autocast else None
    s["x"] = normal(*shape, width, dtype=torch.float32 if autocast and kind != "stack" else dtype)
    if kind != "linear_bwd":
        s["x"].requires_grad_()
    # under autocast a layer's output, and so its upstream gradient, comes in the autocast dtype
    s["g"] = normal(*shape, n_out, scale=case["g_scale"], dtype=s["autocast"] if autocast and kind != "stack" else dtype)
    return s


def run(s):
    case, x, g = s["case"], s["x"], s["g"]
    if case["kind"] == "linear_bwd":
        noise = core.NoiseSpec(std=core.noise_std(case["noise"], case["b"]), seed=_NOISE_KEY, param_id=1, step=1)
        dw, norms, factors = core.dp_linear_weight_grad(x, g, 1.0, 1.0, batch_divisor=case["b"], noise=noise,
                                                        out_dtype=torch.float32, return_norms=True)
        return {"dw": dw, "norms": norms, "factors": factors, "dx": core.linear_input_grad(g, s["weight"])}
    layer = s["layer"]
    layer.zero_grad(set_to_none=True)
    x.grad = None
    if s["autocast"] is not None:
        with torch.autocast("cuda", dtype=s["autocast"]):
            y = layer(x)
    else:
        y = layer(x)
    y.backward(g)
    return {"y": y.detach(), "dx": x.grad, "grads": {n: p.grad for n, p in layer.named_parameters()}}


# ---- what a pass cannot do without -------------------------------------------------------------------
def work(case):
    """Inputs read once, outputs written once; the multiply-adds of the layer's products (forward, input
    gradient, weight gradient).  The per-sample norms, for which no cheaper rule is known than a further
    contraction, are left out."""
    kind = case["kind"]
    if kind == "stack":
        b, t, d, n = case["b"], case["t"], case["width"], case["blocks"]
        rows = b * t
        params = n * (12 * d * d + 13 * d)
        attention = 3.5 * 4.0 * b * t * t * d / 2        # causal; the backward is 2.5 forwards
        return {"bytes": 4.0 * (4 * rows * d + 2 * params), "flops": n * (6.0 * rows * 12 * d * d + attention)}
    if kind == "layernorm":
        elt = 4 if case["dtype"] == "fp32" else 2
        rows, d = case["b"] * case["t"], case["d"]
        return {"bytes": float(elt * (4 * rows * d + 4 * d)), "flops": 16.0 * rows * d}
    rows = case["b"] * max(case["t"], 1)
    n_in, n_out = case["n_in"], case["n_out"]
    elt = 4 if case["dtype"] == "fp32" else 2
    act = 4 if case["autocast"] else elt                 # the layer input and its gradient
    par = 4 if case["autocast"] else elt
    bias = 2 * n_out if case["bias"] else 0
    if kind == "linear_bwd":
        return {"bytes": float(elt * rows * (2 * n_in + n_out) + (elt + 4) * n_in * n_out), "flops": 4.0 * rows * n_in * n_out}
    return {"bytes": float(2 * act * rows * n_in + 2 * elt * rows * n_out + par * (2 * n_in * n_out + bias)),
            "flops": 6.0 * rows * n_in * n_out}


def tolerance(case):
    """About four times the relative error seen against a float64 evaluation of the same inputs: fp32 4.5e-6
    (three bf16 products per fp32 one), bf16 1.7e-3 to 2.3e-3 (rounding of the results, of clipped rows and of
    bias terms), fp16 up to 1.9e-3 (bias gradients reach its subnormal range); for the stack, where roundings
    pass through several layers, 4.5e-3 against the same model with its plain products left to torch."""
    if case["kind"] == "stack":
        return {"rel": 2e-2}
    return {"rel": {"fp32": 2e-5, "bf16": 1e-2, "fp16": 8e-3}[case["dtype"]]}
