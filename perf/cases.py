"""Timed workloads of the simulated-arithmetic path, through the package's public entry points.

``listed()`` gives the fixed cases, ``draw(rng)`` more of the same ranges; ``prepare`` makes what a user's program holds
before the call, ``run`` makes one pass, ``work`` counts the bytes and operations a pass cannot do without, ``tolerance``
says how far a correct result may be off and ``exact`` restates the result in 64-bit torch arithmetic.

Every path here is defined down to the bit (each multiply and each add is rounded to a stated format, in a stated
order), so every tolerance is "exact".
"""
from __future__ import annotations

import math

import torch

import mptorch_b200.quant as q
from mptorch_b200 import FloatingPoint
from mptorch_b200.gpt2_block import BlockConfig, QBlock, default_formats

DEV = "cuda"


# ------------------------------------------------------------------------------------------------------- the cases
def _mm(name, m, n, k, add, mul, batch=0, sub=True, sat=False, fma=False, comp=False, rounding="nearest", order="cuda"):
    """One product; ``add`` and ``mul`` are (mantissa, exponent) bits, ``batch`` 0 means a plain matrix product."""
    return {"name": name, "kind": "mm", "batch": batch, "m": m, "n": n, "k": k, "man_add": add[0], "exp_add": add[1],
            "man_mul": mul[0], "exp_mul": mul[1], "sub": sub, "sat": sat, "fma": fma, "comp": comp, "rounding": rounding,
            "order": order}


E4M3, E5M2, E5M10, E8M7 = (3, 4), (2, 5), (10, 5), (7, 8)


def listed():
    return [
        # a probe of the arithmetic as one writes it at a prompt: latency and launches
        _mm("mm_small", 64, 64, 64, E5M10, E4M3),
        # the headline product of the benchmark, the largest case
        _mm("mm_headline", 8192, 8192, 8192, E5M2, E5M2),
        # bfloat16 accumulation of e5m2 products in the CPU path's sequential order
        _mm("mm_bf16_seq", 2048, 2048, 2048, E8M7, E5M2, order="seq"),
        # formats without subnormals (what FloatingPoint gives by default), no extent a multiple of a tile
        _mm("mm_nosub_ragged", 1500, 1111, 1777, E5M10, E4M3, sub=False),
        # Q K^T of an attention layer as a batched product with fused multiply-adds
        _mm("bmm_fma_attention", 1024, 1024, 64, E5M10, E5M10, batch=96, fma=True),
        # stochastic rounding of every product and sum
        _mm("mm_stochastic", 1024, 1024, 1024, E5M10, E4M3, rounding="stochastic"),
        # a training step of a small classifier's first layer (batch 128, 28 x 28 images) with e4m3 signals: host and
        # launch bound
        {"name": "linear_small_train", "kind": "linear", "rows": 128, "n_in": 784, "n_out": 256, "sub": True},
        # one GPT-2-small block, forward and backward, batch 8 x 1024 tokens (e5m10 sums, e4m3 products)
        {"name": "block_train", "kind": "block", "batch": 8, "seq": 1024, "d": 768, "heads": 12, "mlp": 3072, "sub": True},
        # attention probabilities of that block, forward and backward
        {"name": "softmax_train", "kind": "softmax", "rows": 98304, "cols": 1024, "man": 10, "exp": 5, "sub": True},
        # its layer normalisation, forward and backward with parameter gradients
        {"name": "layernorm_train", "kind": "layernorm", "rows": 8192, "cols": 768, "man": 10, "exp": 5, "sub": True},
        # a 3 x 3 convolution layer of a residual network, forward and backward
        {"name": "conv_train", "kind": "conv", "batch": 64, "c_in": 64, "c_out": 64, "size": 56, "ksize": 3, "stride": 1,
         "sub": True},
        # the elementwise quantizer on a weight-sized tensor with an odd element count
        {"name": "quantize_e4m3", "kind": "quantize", "n": (1 << 26) + 3, "man": 3, "exp": 4, "sub": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mm"] * 7 + ["linear", "block", "softmax", "layernorm", "conv", "quantize"])
    sub = rng.random() < 0.6
    if kind == "mm":
        while True:
            m, n, k = (_log_int(rng, 16, 4096) for _ in range(3))
            batch = rng.choice([0, 0, 0, _log_int(rng, 2, 96)])
            if rng.random() < 0.5:
                m, n, k = ((v + 7) // 8 * 8 for v in (m, n, k))
            if max(batch, 1) * m * n * k <= 1 << 35:
                break
        add, mul = rng.choice([(E5M10, E4M3), (E5M10, E5M2), (E8M7, E5M2), (E8M7, E4M3), (E5M2, E5M2), (E5M10, E5M10), (E8M7, E8M7)])
        form = rng.choice(["plain", "plain", "plain", "plain", "fma", "comp", "stochastic"])
        c = _mm("", m, n, k, add, add if form == "fma" else mul, batch, sub, rng.random() < 0.2, form == "fma", form == "comp",
                "stochastic" if form == "stochastic" else "nearest", rng.choice(["cuda", "cuda", "seq"]))
        del c["name"]
        return c
    if kind == "linear":
        return {"kind": kind, "rows": _log_int(rng, 16, 2048), "n_in": _log_int(rng, 32, 2048), "n_out": _log_int(rng, 10, 2048), "sub": sub}
    if kind == "block":
        heads = rng.choice([2, 4, 6])
        return {"kind": kind, "batch": rng.choice([1, 2, 3]), "seq": _log_int(rng, 64, 1024), "d": 64 * heads, "heads": heads,
                "mlp": 256 * heads, "sub": sub}
    if kind in ("softmax", "layernorm"):
        cols = rng.choice([64, 256, 512, 768, 1024, _log_int(rng, 33, 1500)])
        man, exp = rng.choice([E5M10, E8M7])
        return {"kind": kind, "rows": _log_int(rng, 64, 8192 if kind == "layernorm" else 32768), "cols": cols, "man": man, "exp": exp, "sub": sub}
    if kind == "conv":
        return {"kind": kind, "batch": rng.choice([1, 4, 16]), "c_in": rng.choice([3, 16, 32, 64]), "c_out": rng.choice([10, 16, 32, 64]),
                "size": rng.choice([7, 14, 28, 32, 56]), "ksize": rng.choice([1, 3, 5]), "stride": rng.choice([1, 1, 2]), "sub": sub}
    man, exp = rng.choice([E4M3, E5M2, E5M10, E8M7])
    return {"kind": kind, "n": _log_int(rng, 1000, 1 << 26), "man": man, "exp": exp, "sub": sub}


# ------------------------------------------------------------------------------------------------- inputs of a case
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape):
    return torch.randn(*shape, device=DEV, generator=g)


def _formats(sub, signals=False):
    add, mul = FloatingPoint(5, 10, sub, False), FloatingPoint(4, 3, sub, False)
    kw = {}
    if signals:       # layers whose weights, inputs and gradients are e4m3 as well
        s = (FloatingPoint(4, 3, sub, True), "nearest")
        kw = dict(weight_quant=s, input_quant=s, grad_quant=s)
    return q.QAffineFormats(fwd_mac=(add, mul), bwd_mac=(add, mul), **kw)


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind == "mm":
        lead = (case["batch"],) if case["batch"] else ()
        return {"case": case, "seed": seed, "a": _randn(g, *lead, case["m"], case["k"]), "b": _randn(g, *lead, case["k"], case["n"])}
    if kind == "quantize":
        x = _randn(g, case["n"])
        return {"case": case, "x": x.mul_(torch.pow(2.0, 6 * torch.rand(case["n"], device=DEV, generator=g) - 4))}
    st = {"case": case}
    if kind == "linear":
        layer = q.QLinear(case["n_in"], case["n_out"], _formats(case["sub"], True)).to(DEV)
        with torch.no_grad():
            layer.weight.copy_(_randn(g, case["n_out"], case["n_in"]) / math.sqrt(case["n_in"]))
            layer.bias.copy_(0.1 * _randn(g, case["n_out"]))
        st.update(layer=layer, x=_randn(g, case["rows"], case["n_in"]), gy=_randn(g, case["rows"], case["n_out"]))
    elif kind == "block":
        cfg = BlockConfig(case["d"], case["heads"], case["mlp"], 512, case["seq"])
        layer = QBlock(cfg, default_formats(FloatingPoint(5, 10, case["sub"], False), FloatingPoint(4, 3, case["sub"], False))).to(DEV)
        with torch.no_grad():
            for p in layer.parameters():
                if p.dim() == 2:
                    p.copy_(0.02 * _randn(g, *p.shape))
        st.update(layer=layer, x=_randn(g, case["batch"], case["seq"], case["d"]), gy=_randn(g, case["batch"], case["seq"], case["d"]))
    elif kind == "softmax":
        f = FloatingPoint(case["exp"], case["man"], case["sub"], False)
        layer = q.QSoftmax(-1, q.QSoftmaxFormats(fwd_off=f, fwd_exp=f, fwd_acc=f, bwd_add=f, bwd_mul=f))
        st.update(layer=layer, x=3 * _randn(g, case["rows"], case["cols"]), gy=_randn(g, case["rows"], case["cols"]))
    elif kind == "layernorm":
        f = FloatingPoint(case["exp"], case["man"], case["sub"], False)
        layer = q.QLayerNorm(case["cols"], q.QLayerNormFormats(f, f, f, f, f, f, f)).to(DEV)
        with torch.no_grad():
            layer.weight.copy_(1 + 0.1 * _randn(g, case["cols"]))
            layer.bias.copy_(0.1 * _randn(g, case["cols"]))
        st.update(layer=layer, x=2 * _randn(g, case["rows"], case["cols"]) + 0.5, gy=_randn(g, case["rows"], case["cols"]))
    else:
        k = case["ksize"]
        layer = q.QConv2d(case["c_in"], case["c_out"], k, _formats(case["sub"]), stride=case["stride"], padding=k // 2).to(DEV)
        out = (case["size"] + 2 * (k // 2) - k) // case["stride"] + 1
        with torch.no_grad():
            layer.weight.copy_(_randn(g, *layer.weight.shape) / math.sqrt(case["c_in"] * k * k))
            layer.bias.copy_(0.1 * _randn(g, case["c_out"]))
        st.update(layer=layer, x=_randn(g, case["batch"], case["c_in"], case["size"], case["size"]),
                  gy=_randn(g, case["batch"], case["c_out"], out, out))
    st["x"].requires_grad_(True)
    return st


# ------------------------------------------------------------------------------------------------------ one pass
def run(state):
    c = state["case"]
    if c["kind"] == "mm":
        if c["rounding"] == "stochastic":
            torch.manual_seed(state["seed"])            # the random words are part of the result
        fn = q.float_bmm if c["batch"] else q.float_mm
        with q.orders(accum=c["order"]):
            return fn(state["a"], state["b"], c["man_add"], c["exp_add"], c["man_mul"], c["exp_mul"], rounding=c["rounding"],
                      fma=c["fma"], subnormals=c["sub"], saturate=c["sat"], compensated=c["comp"])
    if c["kind"] == "quantize":
        return q.float_quantize(state["x"], c["exp"], c["man"], rounding="nearest", subnormals=c["sub"], saturate=True)
    layer, x = state["layer"], state["x"]
    x.grad = None
    layer.zero_grad(set_to_none=True)
    y = layer(x)
    y.backward(state["gy"])
    return [y.detach(), x.grad] + [p.grad for p in layer.parameters()]


# ------------------------------------------------------------------------------------------- what a pass cannot avoid
def work(case):
    kind = case["kind"]
    if kind == "mm":
        b, m, n, k = max(case["batch"], 1), case["m"], case["n"], case["k"]
        return {"bytes": 4 * b * (m * k + k * n + m * n), "flops": 2 * b * m * n * k}
    if kind == "quantize":
        return {"bytes": 8 * case["n"], "flops": 0}
    if kind == "linear":
        r, i, o = case["rows"], case["n_in"], case["n_out"]
        return {"bytes": 4 * (2 * r * i + 2 * i * o + 2 * r * o + 2 * o), "flops": 6 * r * i * o}
    if kind == "block":
        b, t, d, f = case["batch"], case["seq"], case["d"], case["mlp"]
        params = 4 * d * d + 2 * d * f + 9 * d + f
        macs = b * t * (4 * d * d + 2 * d * f) + 2 * b * t * t * d
        return {"bytes": 4 * (4 * b * t * d + 2 * params), "flops": 6 * macs}
    if kind == "conv":
        k, s = case["ksize"], case["size"]
        o = (s + 2 * (k // 2) - k) // case["stride"] + 1
        nx, ny = case["batch"] * case["c_in"] * s * s, case["batch"] * case["c_out"] * o * o
        nw = case["c_in"] * case["c_out"] * k * k
        return {"bytes": 4 * (2 * nx + 2 * ny + 2 * nw + 2 * case["c_out"]), "flops": 6 * case["batch"] * o * o * nw}
    e = case["rows"] * case["cols"]      # softmax, layernorm: input, output, gradient in, gradient out
    return {"bytes": 16 * e + (16 * case["cols"] if kind == "layernorm" else 0), "flops": 0}


def tolerance(case):
    return "exact"


# ------------------------------------------------------------------------------------------- 64-bit restatements
def _pow2(e):
    return ((e + 1023) << 52).view(torch.float64)


def _round(x, man, exp, sub, sat):
    """A float64 tensor of float32 values rounded to nearest even in the (exp, man) format."""
    if man >= 23 and exp >= 8:
        return x
    min_exp, max_exp = 2 - (1 << (exp - 1)), (1 << (exp - 1)) - 1
    bits = x.view(torch.int64)
    e = ((bits >> 52) & 0x7FF) - 1023
    quantum = _pow2((e.clamp(min=min_exp) if sub else e.clamp(min=-1000)) - man)
    y = torch.round(x / quantum) * quantum
    if not sub:     # below the smallest normal: that value if the result is in the binade under it and x past its middle, else 0
        low = 2.0 ** min_exp
        up = (y.abs() >= low / 2) & ((bits & 0xFFFFFFFFFFFFF) > (1 << 51))
        y = torch.where(y.abs() < low, torch.where(up, torch.copysign(torch.full_like(y, low), x), torch.zeros_like(y)), y)
    top = (2.0 - 2.0 ** -man) * 2.0 ** max_exp
    over = torch.copysign(torch.full_like(y, top if sat else math.inf), x)
    return torch.where((y.abs() > top) & x.isfinite(), over, y)


def _exact_mm(case, seed):
    st = prepare(case, seed)
    a, b = st["a"].double(), st["b"].double()
    m, n, k = case["m"], case["n"], case["k"]
    # about 20 passes over the 8-byte outputs per step
    if case["rounding"] != "nearest" or case["comp"] or max(case["batch"], 1) * m * n * k > 1 << 34 or k > 6000:
        return None

    def f32(v):
        return v.float().double()

    def add(acc, v):
        return _round(f32(acc + v), case["man_add"], case["exp_add"], case["sub"], case["sat"])

    def step(acc, i):
        p = a[..., :, i, None] * b[..., None, i, :]
        if case["fma"]:
            return add(acc, p)
        return add(acc, _round(f32(p), case["man_mul"], case["exp_mul"], case["sub"], case["sat"]))

    zero = torch.zeros(*a.shape[:-1], n, dtype=torch.float64, device=DEV)
    out = zero
    if case["order"] == "seq":
        for i in range(k):
            out = step(out, i)
        return out
    for k0 in range(0, k, 8):
        inner = zero
        for i in range(k0, min(k, k0 + 8)):
            inner = step(inner, i)
        out = add(out, inner)
    return out


def exact(case, seed):
    """Products and quantizers: the stated roundings in the stated order.  Softmax and layer normalisation: the
    real-number function they approximate (their distance from it is that of the formats).  None for the rest: e4m3
    products flush most of a gradient, so no real-number counterpart is near, nor is there one for a parameter
    gradient summed over thousands of rows in 8 to 11 bits."""
    kind = case["kind"]
    if kind == "mm":
        return _exact_mm(case, seed)
    if kind not in ("quantize", "softmax", "layernorm"):
        return None
    st = prepare(case, seed)
    if kind == "quantize":
        return _round(st["x"].double(), case["man"], case["exp"], case["sub"], True)
    x = st["x"].detach().double().requires_grad_(True)
    if kind == "softmax":
        y = torch.softmax(x, -1)
    else:
        y = torch.nn.functional.layer_norm(x, (case["cols"],), *[p.detach().double() for p in st["layer"].parameters()], 1e-5)
    y.backward(st["gy"].double())
    return [y.detach(), x.grad] + [None] * (2 if kind == "layernorm" else 0)
