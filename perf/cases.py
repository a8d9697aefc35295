"""The work a training or sampling program has this package do, as cases that can be timed.

Every case is one pass through the package's public entry points. ``listed()`` names the cases, ``draw()`` gives
more of the same ranges. Sizes follow the model the package is built for (width 2048, MLP 8192, 16 heads of 128,
512 text tokens of width 1024, 1024 to 4096 image tokens a sample, 1 to 8 samples) and reach down to single small
samples and up to the full batch; image sizes whose token count is no multiple of the kernels' tiles are among them.
"""
from __future__ import annotations

import math

import torch

from anima_trainer_sm120_b200 import (adaln_kernel, fp8_quant, lokr_patch, mlp_patch, mxfp8_gemm, qk_norm_rope, tlokr)
from anima_trainer_sm120_b200.anima_dit import AnimaConfig, GPT2FeedForward
from anima_trainer_sm120_b200.lokr import LokrModule, LokrNetwork
from anima_trainer_sm120_b200.train_step import StepConfig, Trainer

BF16 = torch.bfloat16
RANK = 128
LR = 1e-9      # factors move between passes, as in training, without leaving the distribution they start from


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # k / v projection of one sample's text tokens: the smallest adapted linear, bound by launches
        dict(name="lokr-text-1x512", kind="lokr", batch=1, tokens=512, d_in=1024, d_out=2048, bias=False, fp32=True),
        # an image bucket of 36 x 56 tokens, two samples, a fused qkv width, bias, adapters kept in bf16
        dict(name="lokr-odd-2x2016", kind="lokr", batch=2, tokens=2016, d_in=2048, d_out=6144, bias=True, fp32=False),
        # the largest adapted linear at the full batch
        dict(name="lokr-8x4096", kind="lokr", batch=8, tokens=4096, d_in=2048, d_out=8192, bias=False, fp32=True),
        # the adapted MLP (two linears and the GELU between them) of two samples
        dict(name="mlp-2x4096", kind="mlp", batch=2, tokens=4096, dim=2048, hidden=8192),
        # self-attention's frozen q / k / v while sampling one image: forward only
        dict(name="frozen-sample-1x4096", kind="frozen", batch=1, tokens=4096, d_in=2048, d_out=2048, grad=False),
        # the same projections in a training step at the full batch: forward and input gradient
        dict(name="frozen-train-8x4096", kind="frozen", batch=8, tokens=4096, d_in=2048, d_out=2048, grad=True),
        # quantise and multiply by hand, rows that fill no tile
        dict(name="matmul-1000", kind="matmul", rows=1000, d_in=8192, d_out=2048),
        # timestep-aware adapters of one block (cross-attention's q, k, v, o and the MLP) at the full batch
        dict(name="tlokr-8x4096", kind="tlokr", batch=8, tokens=4096, text=512, dim=2048),
        # modulation and gated residuals of one block, as the quantised training step runs them
        dict(name="adaln-8x4096", kind="adaln", batch=8, tokens=4096, dim=2048, operand=True),
        # the same for one small image (30 x 40 tokens) and bf16 linears behind it
        dict(name="adaln-1x1200", kind="adaln", batch=1, tokens=1200, dim=2048, operand=False),
        # RMSNorm and rotary embedding of q and k
        dict(name="qknorm-8x4096", kind="qknorm", batch=8, tokens=4096, heads=16),
        # a whole optimizer step (two checkpointed blocks, one 512 x 512 image)
        dict(name="step-1x32x32", kind="step", batch=1, high=32, wide=32, text=512, dim=2048, variant="lokr"),
    ]


def _log(rng, lo, hi, multiple):
    """A whole multiple of ``multiple`` in [lo, hi], uniform over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, round(v / multiple) * multiple))


def draw(rng):
    kind = rng.choice(["lokr", "lokr", "mlp", "frozen", "frozen", "matmul", "tlokr", "adaln", "adaln", "qknorm", "step"])
    batch = rng.choice([1, 1, 2, 3, 4, 8])
    if kind == "lokr":
        return dict(kind=kind, batch=batch, tokens=_log(rng, 32, 4096, 32), d_in=_log(rng, 256, 2048, 64),
                    d_out=_log(rng, 256, 8192, 64), bias=rng.random() < 0.3, fp32=rng.random() < 0.7)
    if kind == "mlp":
        dim = _log(rng, 512, 2048, 128)
        return dict(kind=kind, batch=rng.choice([1, 2, 3, 4]), tokens=_log(rng, 64, 4096, 32), dim=dim, hidden=4 * dim)
    if kind == "frozen":
        return dict(kind=kind, batch=batch, tokens=_log(rng, 32, 4096, 16), d_in=_log(rng, 256, 2048, 64),
                    d_out=_log(rng, 256, 2048, 64), grad=rng.random() < 0.6)
    if kind == "matmul":
        return dict(kind=kind, rows=_log(rng, 16, 32768, 1), d_in=_log(rng, 256, 8192, 32), d_out=_log(rng, 256, 8192, 32))
    if kind == "tlokr":
        return dict(kind=kind, batch=rng.choice([1, 2, 4]), tokens=_log(rng, 256, 4096, rng.choice([32, 128])),
                    text=rng.choice([128, 256, 512]), dim=rng.choice([1024, 1536, 2048]))
    if kind == "adaln":
        return dict(kind=kind, batch=batch, tokens=_log(rng, 64, 4096, rng.choice([8, 128])), dim=_log(rng, 512, 2560, 128),
                    operand=rng.random() < 0.6)
    if kind == "qknorm":
        return dict(kind=kind, batch=batch, tokens=_log(rng, 64, 4096, 1), heads=rng.choice([8, 12, 16]))
    return dict(kind=kind, batch=rng.choice([1, 2, 4]), high=rng.choice([16, 24, 32, 40]), wide=rng.choice([16, 32, 48]),
                text=rng.choice([256, 512]), dim=rng.choice([1024, 2048]), variant=rng.choice(["lokr", "tlokr"]))


# ------------------------------------------------------------------------------------------------ states
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(g, *shape, std=1.0, dtype=BF16):
    return (torch.randn(*shape, device="cuda", generator=g) * std).to(dtype)


def _activations(g, *shape):
    """~N(0, 1) with one channel in a thousand scaled by 50, as the activations of such models have."""
    x = torch.randn(*shape, device="cuda", generator=g)
    hot = torch.rand(shape[-1], device="cuda", generator=g) < 1e-3
    return torch.where(hot, x * 50.0, x).to(BF16)


def _linear(g, d_in, d_out):
    lin = torch.nn.Linear(d_in, d_out, bias=False, device="cuda", dtype=BF16).requires_grad_(False)
    lin.weight.copy_(_normal(g, d_out, d_in, std=0.02))
    return lin


def _adapted(g, linears, variant):
    """Adapters in mid-training around ``linears``, hooked in as ``attach_lokr`` does."""
    net = LokrNetwork([LokrModule("lokr_%d" % i, l, lora_dim=RANK, alpha=RANK, factor=8) for i, l in enumerate(linears)])
    lokr_patch.install()
    if variant == "tlokr":
        tlokr.convert_network(net, rank=RANK, min_rank_ratio=0.5)
    net.apply_to()
    for p in net.parameters():
        p.data.copy_(_normal(g, *p.shape, std=0.1 if p.shape == (8, 8) else 0.02, dtype=torch.float32))
    if variant == "tlokr":
        fp8_quant.quantize_tlokr_base_weights(net)
    else:
        lokr_patch.enable_fp8(net)
    return net


def _mlp(g, dim, hidden):
    mlp = GPT2FeedForward(AnimaConfig(dim=64, mlp_dim=64))
    mlp.layer1, mlp.layer2 = _linear(g, dim, hidden), _linear(g, hidden, dim)
    mlp_patch.install(GPT2FeedForward)
    return mlp


def prepare(case, seed):
    c, g = case, _gen(seed)
    s = dict(case)
    kind = c["kind"]
    if kind == "lokr":
        dt = torch.float32 if c["fp32"] else BF16
        s["x"] = _activations(g, c["batch"], c["tokens"], c["d_in"]).requires_grad_(True)
        s["gy"] = _normal(g, c["batch"], c["tokens"], c["d_out"])
        s["W"] = _normal(g, c["d_out"], c["d_in"], std=0.02)
        s["b"] = _normal(g, c["d_out"], std=0.1) if c["bias"] else None
        s["w1"] = _normal(g, 8, 8, std=0.1, dtype=dt).requires_grad_(True)
        s["w2"] = _normal(g, c["d_out"] // 8, c["d_in"] // 8, std=0.02, dtype=dt).requires_grad_(True)
    elif kind == "mlp":
        s["mlp"] = _mlp(g, c["dim"], c["hidden"])
        s["net"] = _adapted(g, [s["mlp"].layer1, s["mlp"].layer2], "lokr")
        s["params"] = list(s["net"].parameters())
        s["x"] = _normal(g, c["batch"], c["tokens"], c["dim"]).requires_grad_(True)
        s["gy"] = _normal(g, c["batch"], c["tokens"], c["dim"])
    elif kind == "frozen":
        s["W"] = [_normal(g, c["d_out"], c["d_in"], std=0.02) for _ in range(3)]
        s["Wq"] = [fp8_quant.quantize_weight(W) for W in s["W"]]
        s["x"] = _activations(g, c["batch"], c["tokens"], c["d_in"]).requires_grad_(c["grad"])
        if c["grad"]:
            s["gy"] = [_normal(g, c["batch"], c["tokens"], c["d_out"]) for _ in range(3)]
    elif kind == "matmul":
        s["x"] = _activations(g, c["rows"], c["d_in"])
        s["Wq"] = mxfp8_gemm.quantize_weight_for_lhs(_normal(g, c["d_out"], c["d_in"], std=0.02))
    elif kind == "tlokr":
        dim = c["dim"]
        s["attn"] = [_linear(g, dim, dim), _linear(g, 1024, dim), _linear(g, 1024, dim), _linear(g, dim, dim)]
        s["mlp"] = _mlp(g, dim, 4 * dim)
        s["net"] = _adapted(g, s["attn"] + [s["mlp"].layer1, s["mlp"].layer2], "tlokr")
        s["params"] = list(s["net"].parameters())
        s["t"] = torch.rand(c["batch"], device="cuda", generator=g)
        img, txt = (c["batch"], c["tokens"], dim), (c["batch"], c["text"], 1024)
        s["x"] = [_normal(g, *img).requires_grad_(True) for _ in range(3)]      # inputs of q, o and the MLP
        s["ctx"] = _normal(g, *txt)
        s["gy"] = [_normal(g, c["batch"], n, dim) for n in (c["tokens"], c["text"], c["text"], c["tokens"], c["tokens"])]
    elif kind == "adaln":
        adaln_kernel.emit_row_operand(c["operand"])
        shape, mod = (c["batch"], 1, 1, c["tokens"], c["dim"]), (c["batch"], 1, 1, 1, c["dim"])
        s["x"], s["a"], s["m"] = (_normal(g, *shape).requires_grad_(True) for _ in range(3))
        s["mods"] = [_normal(g, *mod, std=0.1).requires_grad_(True) for _ in range(6)]
        s["gn"], s["ga"], s["go"] = (_normal(g, *shape) for _ in range(3))
    elif kind == "qknorm":
        shape = (c["batch"], c["tokens"], c["heads"], 128)
        s["q"], s["k"] = (_normal(g, *shape).requires_grad_(True) for _ in range(2))
        s["gq"], s["gk"] = (_normal(g, *shape) for _ in range(2))
        s["w"] = [(1.0 + _normal(g, 128, std=0.1, dtype=torch.float32)).to(BF16) for _ in range(2)]
        ang = torch.rand(c["tokens"], 1, 1, 64, device="cuda", generator=g) * 6.28
        s["tables"] = qk_norm_rope.rope_tables(torch.cat([ang, ang], dim=-1))
    elif kind == "step":
        cfg = AnimaConfig(depth=2, dim=c["dim"], heads=c["dim"] // 128, mlp_dim=4 * c["dim"])
        with torch.device("cuda"):
            tr = Trainer(cfg, StepConfig(precision="mxfp8", variant=c["variant"], seed=seed), torch.device("cuda", 0))
        for p in tr.params:                       # adapters in mid-training, not at their zero start
            p.data.copy_(_normal(g, *p.shape, std=0.1 if p.shape == (8, 8) else 0.02, dtype=torch.float32))
        s["trainer"], s["noise"] = tr, seed + 1
        s["latents"] = _normal(g, c["batch"], 16, 1, 2 * c["high"], 2 * c["wide"])
        s["ctx"] = _normal(g, c["batch"], c["text"], cfg.context_dim)
    else:
        raise ValueError("unknown kind %r" % kind)
    return s


# ------------------------------------------------------------------------------------------------ one pass
def _sgd(params, grads):
    torch._foreach_add_(list(params), list(grads), alpha=-LR)


def run(s):
    kind = s["kind"]
    fp8_quant.clear_activation_memo()          # a training step's activations are new tensors
    if kind == "lokr":
        y = fp8_quant.lokr_linear_fused(s["x"], s["W"], s["b"], s["w1"], s["w2"], 1.0)
        return (y, *torch.autograd.grad(y, (s["x"], s["w1"], s["w2"]), s["gy"]))
    if kind == "mlp":
        y = s["mlp"](s["x"])
        gx, *gp = torch.autograd.grad(y, [s["x"], *s["params"]], s["gy"])
        with torch.no_grad():
            _sgd(s["params"], gp)
        return (y, gx, *gp, *s["params"])
    if kind == "frozen":
        with torch.set_grad_enabled(s["grad"]):
            ys = [fp8_quant.mxfp8_frozen_linear(s["x"], q, W) for q, W in zip(s["Wq"], s["W"])]
        if not s["grad"]:
            return ys
        return (*ys, *torch.autograd.grad(ys, s["x"], s["gy"]))
    if kind == "matmul":
        xq = mxfp8_gemm.quantize_rowwise(s["x"])
        y = mxfp8_gemm.mxfp8_matmul(xq, s["Wq"].data, s["Wq"].scales, s["rows"], s["d_out"], s["d_in"], 1, s["d_in"],
                                    B_tiled=s["Wq"].tiled)
        return xq.data, xq.scales, y
    if kind == "tlokr":
        q, k, v, o = s["attn"]
        xq, xo, xm = s["x"]
        tlokr.set_timestep(s["t"])
        try:
            ys = [q(xq), k(s["ctx"]), v(s["ctx"]), o(xo), s["mlp"](xm)]
            grads = torch.autograd.grad(ys, [xq, xo, xm, *s["params"]], s["gy"])
        finally:
            tlokr.clear_timestep()
        with torch.no_grad():
            _sgd(s["params"], grads[3:])
        return (*ys, *grads, *s["params"])
    if kind == "adaln":
        g0, sc0, sh0, g1, sc1, sh1 = s["mods"]
        n0 = adaln_kernel.fused_adaln(s["x"], sc0, sh0, 1e-6)
        x1, n1 = adaln_kernel.fused_gated_add_adaln(s["x"], g0, s["a"], sc1, sh1, 1e-6)
        out = adaln_kernel.fused_gated_add(x1, g1, s["m"])
        grads = torch.autograd.grad([n0, n1, out], [s["x"], s["a"], s["m"], *s["mods"]], [s["gn"], s["ga"], s["go"]])
        ops = ()
        if s["operand"] and (s["batch"] * s["tokens"]) % 128 == 0:       # what the linear behind it reads
            op = fp8_quant.quantize_activation(n1, colwise=False)[0]
            ops = (op.codes, op.scales)
        return (n0, x1, n1, out, *grads, *ops)
    if kind == "qknorm":
        cos, sin = s["tables"]
        q = qk_norm_rope.FusedRMSNormRoPE.apply(s["q"], s["w"][0], cos, sin, 1e-6)
        k = qk_norm_rope.FusedRMSNormRoPE.apply(s["k"], s["w"][1], cos, sin, 1e-6)
        return (q, k, *torch.autograd.grad([q, k], [s["q"], s["k"]], [s["gq"], s["gk"]]))
    tr = s["trainer"]
    loss = tr.step(s["latents"], s["ctx"], s["noise"])
    return (loss, tr.flat_grad, *tr.params)


# ------------------------------------------------------------------------------------------------ what a pass needs
def work(case):
    c, kind = case, case["kind"]
    if kind == "matmul":
        m, n, k = c["rows"], c["d_out"], c["d_in"]
        return {"bytes": 3.03 * m * k + 1.03 * n * k + 2 * m * n, "flops": 2.0 * m * n * k}
    rows = c["batch"] * c.get("tokens", 0)
    if kind == "lokr":
        n, k = c["d_out"], c["d_in"]
        return {"bytes": 4.0 * rows * (n + k) + 2 * n * k + n * k / 8, "flops": 6.0 * rows * n * k}
    if kind == "mlp":
        d, h = c["dim"], c["hidden"]
        return {"bytes": 8.0 * rows * d + 4 * d * h + 4 * d * h / 8, "flops": 12.0 * rows * d * h}
    if kind == "frozen":
        n, k, both = c["d_out"], c["d_in"], 2 if c["grad"] else 1
        return {"bytes": both * (2.0 * rows * (k + 3 * n) + 3 * 1.03 * n * k), "flops": both * 6.0 * rows * n * k}
    if kind == "tlokr":
        d, t = c["dim"], c["batch"] * c["text"]
        pairs = [(rows, d, d), (rows, d, d), (rows, d, 4 * d), (rows, 4 * d, d), (t, 1024, d), (t, 1024, d)]
        flops = sum((4.0 if m == rows else 2.0) * m * k * n + RANK * m * (6.0 * k + 6.0 * n) for m, k, n in pairs)
        return {"bytes": 2.0 * (rows * 12 * d + t * (1024 + 4 * d)) + 2.06 * (10 * d * d + 2048 * d), "flops": flops}
    if kind == "adaln":
        e = float(rows * c["dim"])                # 3 inputs, 4 outputs; 3 gradients in and out, 3 saved activations
        return {"bytes": 2 * e * 16 + (2.06 * e if c["operand"] and rows % 128 == 0 else 0), "flops": 60 * e}
    if kind == "qknorm":
        e = float(rows * c["heads"] * 128)        # forward in and out, backward two in and one out, q and k
        return {"bytes": 2 * 5 * 2 * e, "flops": 40 * e}
    d, rows, t = c["dim"], c["batch"] * c["high"] * c["wide"], c["batch"] * c["text"]
    linear = 16.0 * rows * d * d + 12.0 * rows * d * d + 12.0 * t * 1024 * d + 48.0 * rows * d * d
    attention = 14.0 * rows * d * (c["high"] * c["wide"] + c["text"])
    return {"bytes": 2 * (2.0 * 2 * 16 * d * d + 40.0 * rows * d), "flops": 2 * (linear + attention)}


def tolerance(case):
    # bf16 tensors, and e4m3 codes made from them: a sum that rounds the other way moves a code by one step
    if case["kind"] == "step":
        return {"rel": 2e-2}       # two blocks deep, library attention between them
    if case["kind"] in ("adaln", "qknorm"):
        return {"rel": 5e-3, "differ": 1e-2}
    return {"rel": 1e-2}
