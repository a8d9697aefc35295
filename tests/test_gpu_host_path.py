"""Native autograd nodes: what a pass computes follows from which inputs want a gradient. Every subset of the
gradients, the no-grad forward and the checkpointed form must give the bits of the full pass (same kernels on the
same operands), so the comparisons are exact."""
from __future__ import annotations

import pytest
import torch
from torch.utils.checkpoint import checkpoint

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16
DEV = "cuda"


def _randn(g, *shape, std=1.0, dtype=BF16):
    return (torch.randn(*shape, device=DEV, generator=g) * std).to(dtype)


def _lokr(rows):
    from anima_trainer_sm120_b200.fp8_quant import lokr_linear_fused
    g = torch.Generator(device=DEV).manual_seed(rows)
    W, bias = _randn(g, 512, 256, std=0.05), _randn(g, 512)
    ts = [_randn(g, 1, rows, 256), _randn(g, 8, 8, std=0.1, dtype=torch.float32),
          _randn(g, 64, 32, std=0.1, dtype=torch.float32)]
    return lambda x, w1, w2: lokr_linear_fused(x, W, bias, w1, w2, 0.7), ts, (1, rows, 512)


def _merged(rows):
    from anima_trainer_sm120_b200.fp8_quant import mxfp8_lokr_linear
    g = torch.Generator(device=DEV).manual_seed(rows)
    return (lambda x, W: mxfp8_lokr_linear(x, W)), [_randn(g, rows, 256), _randn(g, 512, 256, std=0.05)], (rows, 512)


def _mlp(rows):
    from anima_trainer_sm120_b200.mlp_patch import LoKrMLPFused
    g = torch.Generator(device=DEV).manual_seed(rows)
    W1, W2 = _randn(g, 512, 256, std=0.05), _randn(g, 256, 512, std=0.05)
    f = lambda *s: _randn(g, *s, std=0.1, dtype=torch.float32)
    ts = [_randn(g, 1, rows, 256), f(8, 8), f(64, 32), f(8, 8), f(32, 64)]
    return (lambda x, a, b, c, d: LoKrMLPFused.apply(x, W1, None, a, b, 0.7, W2, None, c, d, 1.3)), ts, (1, rows, 256)


def _tlokr(rows):
    from anima_trainer_sm120_b200 import tlokr
    from anima_trainer_sm120_b200.fp8_quant import quantize_weight
    g = torch.Generator(device=DEV).manual_seed(rows)
    W = quantize_weight(_randn(g, 1024, 512, std=0.05))
    f = lambda *s: _randn(g, *s, std=0.1, dtype=torch.float32)
    ts = [_randn(g, 2, rows, 512), f(8, 8), f(128, 128), f(128, 64)]
    mask = (torch.arange(128, device=DEV)[None] < torch.tensor([[70], [120]], device=DEV)).to(BF16)
    return (lambda x, w1, a, b: tlokr._MXTLoKrLinear.apply(x, W, None, w1, a, b, mask, 0.5)), ts, (2, rows, 1024)


@pytest.mark.parametrize("make,rows", [(_lokr, 32), (_lokr, 160), (_merged, 96), (_mlp, 64), (_tlokr, 48), (_tlokr, 128)])
def test_every_gradient_subset_and_the_checkpointed_pass_give_the_same_bits(make, rows):
    from anima_trainer_sm120_b200 import fp8_quant
    fn, ts, out_shape = make(rows)
    g = torch.Generator(device=DEV).manual_seed(1)
    gy = _randn(g, *out_shape)

    def go(subset, wrap=None):
        fp8_quant.clear_activation_memo()
        leaves = [t.clone().requires_grad_(i in subset) for i, t in enumerate(ts)]
        y = (wrap or fn)(*leaves)
        if subset:
            y.backward(gy)
        return y.detach(), [t.grad for t in leaves]

    everything = set(range(len(ts)))
    y, grads = go(everything)
    assert y.shape == out_shape and all(g is not None for g in grads)
    for subset in [set(), {0}, everything - {0}, {len(ts) - 1}]:
        y2, some = go(subset)
        assert torch.equal(y2, y)
        for i, (a, b) in enumerate(zip(some, grads)):
            assert (a is None) == (i not in subset)
            assert a is None or torch.equal(a, b)
    with torch.no_grad():
        fp8_quant.clear_activation_memo()
        assert torch.equal(fn(*ts), y)

    def checkpointed(*leaves):
        with fp8_quant.first_pass():
            return checkpoint(fn, *leaves, use_reentrant=False)

    y3, again = go(everything, checkpointed)
    assert torch.equal(y3, y) and all(torch.equal(a, b) for a, b in zip(again, grads))
