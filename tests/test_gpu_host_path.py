"""Native autograd nodes: what a pass computes follows from which inputs want a gradient. Every subset of the
gradients, the no-grad forward and the checkpointed form must give the bits of the full pass (same kernels on the
same operands), so the comparisons are exact."""
from __future__ import annotations

import contextlib

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


def _tlokr_mlp(rows):
    from anima_trainer_sm120_b200 import tlokr
    from anima_trainer_sm120_b200.fp8_quant import quantize_weight
    g = torch.Generator(device=DEV).manual_seed(rows)
    W1, W2 = quantize_weight(_randn(g, 1024, 512, std=0.05)), quantize_weight(_randn(g, 512, 1024, std=0.05))
    f = lambda *s: _randn(g, *s, std=0.1, dtype=torch.float32)
    ts = [_randn(g, 2, rows, 512), f(8, 8), f(128, 128), f(128, 64), f(8, 8), f(64, 128), f(128, 128)]
    return (lambda x, c1, a1, b1, c2, a2, b2: tlokr._MXTLoKrMLP.apply(x, W1, None, c1, a1, b1, None, 0.5, W2, None, c2, a2, b2,
                                                                      None, 0.5)), ts, (2, rows, 512)


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


@pytest.mark.parametrize("make,rows", [(_lokr, 32), (_merged, 96), (_mlp, 64), (_tlokr, 128), (_tlokr_mlp, 128)])
def test_backward_through_a_first_pass_without_a_checkpoint_is_refused(make, rows):
    """Its operands are stand-ins without memory; the refusal comes before the first launch of the node."""
    from anima_trainer_sm120_b200 import fp8_quant
    fn, ts, out_shape = make(rows)
    leaves = [t.clone().requires_grad_() for t in ts]
    fp8_quant.clear_activation_memo()
    with fp8_quant.first_pass():
        y = fn(*leaves)
    with pytest.raises(RuntimeError, match="first_pass"):
        y.backward(torch.ones(out_shape, device=DEV, dtype=BF16))
    assert all(t.grad is None for t in leaves)


def _block_inputs(B, hw, D, mod_grad, chunked):
    g = torch.Generator(device=DEV).manual_seed(hw + D)
    x, sub = (_randn(g, B, 1, hw, 1, D).requires_grad_(True) for _ in range(2))
    if chunked:                               # chunks of one (B, 1, 3 D) tensor, as a modulation MLP returns them
        mods = [m[:, :, None, None, :] for m in (_randn(g, B, 1, 6 * D, std=0.1)).chunk(6, dim=-1)[:4]]
    else:
        mods = [_randn(g, B, 1, 1, 1, D, std=0.1) for _ in range(4)]
    mods = [m.detach().requires_grad_(mod_grad) for m in mods]
    return x, sub, mods, [_randn(g, B, 1, hw, 1, D) for _ in range(3)]


@pytest.mark.parametrize("B,hw,D", [(2, 24, 256), (1, 7, 2048), (3, 130, 264), (2, 16, 4096)])
@pytest.mark.parametrize("mod_grad,chunked", [(True, False), (False, True), (True, True)])
def test_residual_gradient_through_the_modulation_equals_the_separate_sum(B, hw, D, mod_grad, chunked):
    """x feeds a modulation and the gated residual behind it: its gradient is formed in the modulation's backward
    kernel. The same graph with the residual reading an unrelated alias of x adds the two gradients in bf16."""
    from anima_trainer_sm120_b200.adaln_kernel import fused_adaln, fused_gated_add_adaln
    results = []
    for routed in (True, False):
        x, sub, (g0, sc, sh, sc1), (gn, gx, gy) = _block_inputs(B, hw, D, mod_grad, chunked)
        n = fused_adaln(x, sc, sh, 1e-6)
        x_new, y = fused_gated_add_adaln(x if routed else x.view_as(x), g0, sub, sc1, sh, 1e-6)
        mods = [m for m in (g0, sc, sh, sc1) if mod_grad]
        results.append([n.detach(), x_new.detach(), y.detach(),
                        *torch.autograd.grad([n, x_new, y], [x, sub, *mods], [gn, gx, gy])])
    for a, b in zip(*results):
        assert torch.equal(a, b)


@pytest.mark.parametrize("shape", [(1, 2, 1, 1, 256), (1, 1, 1, 1, 512), (2, 256), (512,), (4, 1, 1, 1, 128)])
def test_modulation_of_any_shape_is_read_in_order(shape):
    """As rows of the activation's width, whatever the shape says; its gradient has that shape."""
    from anima_trainer_sm120_b200.adaln_kernel import fused_adaln, fused_gated_add, fused_gated_add_adaln

    def go(as_given):
        x, sub, mods, (gn, gx, gy) = _block_inputs(2, 24, 256, True, False)
        ms = [m.detach().reshape(as_given).requires_grad_() for m in mods]
        outs = [fused_adaln(x, ms[1], ms[2], 1e-6), *fused_gated_add_adaln(x, ms[0], sub, ms[3], ms[2], 1e-6),
                fused_gated_add(x, ms[0], sub)]
        grads = torch.autograd.grad(outs, [x, sub, *ms], [gn, gx, gy, gx])
        assert all(g.shape == as_given for g in grads[2:])
        return [t.detach().reshape(-1) for t in (*outs, *grads)]

    for a, b in zip(go((2, 1, 1, 1, 256)), go(shape)):
        assert torch.equal(a, b)


def test_gradient_of_the_bias_alone():
    from anima_trainer_sm120_b200 import fp8_quant
    g = torch.Generator(device=DEV).manual_seed(7)
    x, W, gy = _randn(g, 64, 256), _randn(g, 512, 256, std=0.05), _randn(g, 64, 512)
    Q, w1, w2 = fp8_quant.quantize_weight(W), _randn(g, 8, 8), _randn(g, 64, 32)
    for call in (lambda b: fp8_quant.lokr_linear_fused(x, W, b, w1, w2, 1.0), lambda b: fp8_quant.mxfp8_lokr_linear(x, W, b),
                 lambda b: fp8_quant.mxfp8_frozen_linear(x, Q, W, b)):
        b = torch.zeros(512, device=DEV, dtype=BF16, requires_grad=True)
        call(b).backward(gy)
        assert torch.equal(b.grad, gy.sum(0))


def test_tlokr_forward_of_a_base_weight_without_its_column_form():
    """quantize_weight(..., with_dgrad=False): enough for a pass that makes no input gradient."""
    from anima_trainer_sm120_b200 import tlokr
    from anima_trainer_sm120_b200.fp8_quant import quantize_weight
    g = torch.Generator(device=DEV).manual_seed(8)
    W = _randn(g, 1024, 512, std=0.05)
    f = lambda *s: _randn(g, *s, std=0.1, dtype=torch.float32).requires_grad_()
    x, factors, gy = _randn(g, 2, 96, 512), [f(8, 8), f(128, 128), f(128, 64)], _randn(g, 2, 96, 1024)
    results = []
    for with_dgrad in (True, False):
        y = tlokr._MXTLoKrLinear.apply(x, quantize_weight(W, with_dgrad=with_dgrad), None, *factors, None, 0.5)
        results.append([y.detach(), *torch.autograd.grad(y, factors, gy)])
    assert all(torch.equal(a, b) for a, b in zip(*results))
    y = tlokr._MXTLoKrLinear.apply(x.clone().requires_grad_(), quantize_weight(W, with_dgrad=False), None, *factors, None, 0.5)
    with pytest.raises(ValueError, match="column form"):
        y.backward(gy)


@pytest.mark.parametrize("which", ["w1", "a", "b", "mask"])
@pytest.mark.parametrize("mask_dtype", [BF16, torch.float32])
def test_tlokr_tensors_changed_in_place_before_backward_are_noticed(which, mask_dtype):
    from anima_trainer_sm120_b200 import tlokr
    from anima_trainer_sm120_b200.fp8_quant import quantize_weight
    g = torch.Generator(device=DEV).manual_seed(9)
    f = lambda *s: _randn(g, *s, std=0.1, dtype=torch.float32).requires_grad_()
    ts = {"w1": f(8, 8), "a": f(128, 128), "b": f(128, 64), "mask": torch.ones(2, 128, device=DEV, dtype=mask_dtype)}
    x, W = _randn(g, 2, 64, 512).requires_grad_(), quantize_weight(_randn(g, 1024, 512, std=0.05))
    y = tlokr._MXTLoKrLinear.apply(x, W, None, ts["w1"], ts["a"], ts["b"], ts["mask"], 0.5)
    with torch.no_grad():
        ts[which].mul_(0.5)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.backward(torch.ones_like(y))


def test_backward_weight_of_the_block_level_frozen_linear_is_a_saved_tensor():
    """W_bwd changed in place, or a second backward through a freed graph, is refused; a retained graph is not."""
    from anima_trainer_sm120_b200 import mxfp8_gemm
    g = torch.Generator(device=DEV).manual_seed(10)
    W, x, gy = _randn(g, 256, 128, std=0.05), _randn(g, 96, 128).requires_grad_(), _randn(g, 96, 256)
    go = lambda: mxfp8_gemm.mxfp8_frozen_linear_triton(x, mxfp8_gemm.quantize_weight_for_lhs(W), W_bwd)
    W_bwd = mxfp8_gemm.quantize_weight_for_dgrad(W)
    y = go()
    first, = torch.autograd.grad(y, x, gy, retain_graph=True)
    again, = torch.autograd.grad(y, x, gy)
    assert torch.equal(first, again)
    with pytest.raises(RuntimeError, match="second time"):
        y.backward(gy)
    y = go()
    W_bwd.data.zero_()
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.backward(gy)


@pytest.mark.parametrize("which", ["lokr W", "frozen W", "mlp W1", "mlp b2", "tlokr mlp b1", "norm weight"])
def test_output_belongs_to_the_graph_of_a_trainable_tensor_without_a_gradient_rule(which):
    """As for any autograd function: backward runs, that tensor's gradient is none, the others are what they are without it."""
    from anima_trainer_sm120_b200 import fp8_quant, tlokr
    from anima_trainer_sm120_b200.fp8_quant import quantize_weight
    from anima_trainer_sm120_b200.mlp_patch import LoKrMLPFused
    from anima_trainer_sm120_b200.qk_norm_rope import FusedRMSNormRoPE
    g = torch.Generator(device=DEV).manual_seed(11)
    W1, W2, x = _randn(g, 512, 256, std=0.05), _randn(g, 256, 512, std=0.05), _randn(g, 1, 64, 256)
    w1, w2, w2t, f = _randn(g, 8, 8), _randn(g, 64, 32), _randn(g, 32, 64), lambda *s: _randn(g, *s, std=0.1)
    a1, b1, a2, b2 = f(64, 128), f(128, 32), f(32, 128), f(128, 64)
    Q1, Q2, heads = quantize_weight(W1), quantize_weight(W2), _randn(g, 1, 16, 2, 128)
    call, t, inp = {
        "lokr W": (lambda x, t: fp8_quant.lokr_linear_fused(x, t, None, w1, w2, 1.0), W1, x),
        "frozen W": (lambda x, t: fp8_quant.mxfp8_frozen_linear(x, Q1, t), W1, x),
        "mlp W1": (lambda x, t: LoKrMLPFused.apply(x, t, None, w1, w2, 1.0, W2, None, w1, w2t, 1.0), W1, x),
        "mlp b2": (lambda x, t: LoKrMLPFused.apply(x, W1, None, w1, w2, 1.0, W2, t, w1, w2t, 1.0), _randn(g, 256), x),
        "tlokr mlp b1": (lambda x, t: tlokr._MXTLoKrMLP.apply(x, Q1, t, w1, a1, b1, None, 0.5, Q2, None, w1, a2, b2, None, 0.5),
                         _randn(g, 512), x),
        "norm weight": (lambda x, t: FusedRMSNormRoPE.apply(x, t, None, None, 1e-6), _randn(g, 128), heads),
    }[which]
    grads = []
    for x_wants in (False, True):
        for t_wants in (False, True):
            xi, ti = inp.clone().requires_grad_(x_wants), t.clone().requires_grad_(t_wants)
            y = call(xi, ti)
            assert y.requires_grad == (x_wants or t_wants)
            if y.requires_grad:
                y.backward(torch.ones_like(y))
                assert ti.grad is None
                grads.append(xi.grad)
    assert grads[0] is None and torch.equal(grads[1], grads[2])


@pytest.mark.parametrize("dtype", [BF16, torch.float32])
@pytest.mark.parametrize("tokens,heads", [(1, 1), (5, 3), (40, 16)])
def test_norm_weight_changed_before_backward(dtype, tokens, heads):
    """A bf16 weight is used as forward read it; an fp32 one is a kept tensor, whose change is refused."""
    from anima_trainer_sm120_b200.qk_norm_rope import FusedRMSNormRoPE
    g = torch.Generator(device=DEV).manual_seed(tokens)
    x, gy = _randn(g, 1, tokens, heads, 128).requires_grad_(), _randn(g, 1, tokens, heads, 128)
    w = (1 + _randn(g, 128, std=0.1, dtype=torch.float32)).to(dtype)
    want, = torch.autograd.grad(FusedRMSNormRoPE.apply(x, w, None, None, 1e-6), x, gy)
    y = FusedRMSNormRoPE.apply(x, w, None, None, 1e-6)
    w.mul_(3)
    if dtype == BF16:
        assert torch.equal(torch.autograd.grad(y, x, gy)[0], want)
    else:
        with pytest.raises(RuntimeError, match="modified by an inplace operation"):
            y.backward(gy)


@pytest.mark.parametrize("chunked", [False, True])
def test_saved_tensors_moved_by_hooks_give_the_same_gradients(chunked):
    """save_on_cpu hands every saved tensor back dense: also the chunks of one modulation tensor, whose rows had a pitch."""
    from anima_trainer_sm120_b200.adaln_kernel import fused_adaln, fused_gated_add, fused_gated_add_adaln
    results = []
    for moved in (False, True):
        x, sub, (g0, sc, sh, sc1), (gn, gx, gy) = _block_inputs(3, 40, 256, True, chunked)
        with torch.autograd.graph.save_on_cpu() if moved else contextlib.nullcontext():
            outs = [fused_adaln(x, sc, sh, 1e-6), *fused_gated_add_adaln(x, g0, sub, sc1, sh, 1e-6),
                    fused_gated_add(x.detach(), g0, sub)]
        results.append(torch.autograd.grad(outs, [x, sub, g0, sc, sh, sc1], [gn, gx, gy, gx]))
    assert all(torch.equal(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("make,rows", [(_lokr, 160), (_merged, 96), (_mlp, 64), (_tlokr, 128), (_tlokr_mlp, 128)])
def test_saved_operands_moved_by_hooks_give_the_same_gradients(make, rows):
    from anima_trainer_sm120_b200 import fp8_quant
    fn, ts, out_shape = make(rows)
    gy = _randn(torch.Generator(device=DEV).manual_seed(1), *out_shape)
    results = []
    for moved in (False, True):
        fp8_quant.clear_activation_memo()
        leaves = [t.clone().requires_grad_() for t in ts]
        with torch.autograd.graph.save_on_cpu() if moved else contextlib.nullcontext():
            y = fn(*leaves)
        results.append(torch.autograd.grad(y, leaves, gy))
    assert all(torch.equal(a, b) for a, b in zip(*results))


class _NoGradient(torch.autograd.Function):
    @staticmethod
    def forward(ctx, t):
        return t.clone()

    @staticmethod
    def backward(ctx, g):
        return None


@pytest.mark.parametrize("used", ["x_new", "y", "neither"])
def test_outputs_without_an_incoming_gradient_count_as_zero(used):
    from anima_trainer_sm120_b200.adaln_kernel import fused_adaln, fused_gated_add_adaln
    results = []
    for explicit in (True, False):
        x, sub, (g0, sc, sh, _), (_, gx, gy) = _block_inputs(2, 24, 256, True, False)
        x_new, y = fused_gated_add_adaln(x, g0, sub, sc, sh, 1e-6)
        zero = torch.zeros_like(gx)
        if explicit:
            outs, gs = [x_new, y], [gx if used == "x_new" else zero, gy if used == "y" else zero]
        elif used == "neither":
            outs, gs = [_NoGradient.apply(y)], [gy]
        else:
            outs, gs = [x_new if used == "x_new" else y], [gx if used == "x_new" else gy]
        results.append(torch.autograd.grad(outs, [x, sub, g0, sc, sh], gs))
    assert all(torch.equal(a, b) for a, b in zip(*results))
    x, _, (_, sc, sh, _), (gn, _, _) = _block_inputs(2, 24, 256, True, False)
    for t in torch.autograd.grad(_NoGradient.apply(fused_adaln(x, sc, sh, 1e-6)), [x, sc, sh], gn):
        assert t.count_nonzero() == 0


def test_modulation_and_residual_can_be_backpropagated_one_after_the_other():
    from anima_trainer_sm120_b200.adaln_kernel import fused_adaln, fused_gated_add
    for order in ((0, 1), (1, 0)):
        grads = []
        for routed in (True, False):
            x, sub, (g0, sc, sh, _), (gn, gx, _) = _block_inputs(2, 24, 256, True, False)
            outs = [fused_adaln(x, sc, sh, 1e-6), fused_gated_add(x if routed else x.view_as(x), g0, sub)]
            for i in order:
                outs[i].backward((gn, gx)[i])
            grads.append([t.grad for t in (x, sub, g0, sc, sh)])
            with pytest.raises(RuntimeError):
                outs[0].backward(gn)                       # its saved tensors are gone, as for any node
        for a, b in zip(*grads):
            assert torch.equal(a, b)


@pytest.mark.parametrize("rows,ks", [(160, (256, 512, 96)), (1000, (256, 256, 256)), (96, (256, 256, 128)), (4096, (2048, 2048, 2048))])
def test_input_gradient_of_frozen_linears_of_one_tensor_is_the_bf16_sum_of_their_own(rows, ks):
    """Each linear rounds its own product to bf16 and autograd adds them in bf16, the one applied last first: the bits of
    that sum, whichever of the outputs are used."""
    from anima_trainer_sm120_b200 import _lib, fp8_quant
    g = torch.Generator(device=DEV).manual_seed(rows)
    d_in = 320
    x = _randn(g, rows, d_in).requires_grad_(True)
    Ws = [_randn(g, k, d_in, std=0.05) for k in ks]
    Qs = [fp8_quant.quantize_weight(W) for W in Ws]
    gys = [_randn(g, rows, k) for k in ks]
    lin = lambda i: fp8_quant.mxfp8_frozen_linear(x, Qs[i], Ws[i])
    single = [torch.autograd.grad(lin(i), x, gys[i])[0] for i in range(3)]
    for used in [[0, 1, 2], [0], [2], [0, 2]]:
        fp8_quant.clear_activation_memo()
        ys = [lin(i) for i in range(3)]
        assert len({y.grad_fn for y in ys}) == 3
        gx, = torch.autograd.grad([ys[i] for i in used], x, [gys[i] for i in used])
        want = single[used[-1]]
        for i in used[-2::-1]:
            want = want + single[i]
        assert torch.equal(gx, want)
    _lib.check_status_word(x.device)


def test_frozen_linear_with_a_trainable_bias_after_another_of_the_same_input_was_consumed():
    from anima_trainer_sm120_b200 import fp8_quant
    g = torch.Generator(device=DEV).manual_seed(6)
    W, bias = _randn(g, 256, 256, std=0.05), _randn(g, 256).requires_grad_(True)
    Q, gy = fp8_quant.quantize_weight(W), _randn(g, 160, 256)
    x = _randn(g, 160, 256).requires_grad_(True)
    q = fp8_quant.mxfp8_frozen_linear(x, Q, W).view(160, 2, 128)       # its node has a consumer now
    k = fp8_quant.mxfp8_frozen_linear(x, Q, W, bias)
    gx, gb = torch.autograd.grad([q, k], [x, bias], [gy.view(160, 2, 128), gy])
    one, = torch.autograd.grad(fp8_quant.mxfp8_frozen_linear(x, Q, W), x, gy)
    assert torch.equal(gx, one + one) and torch.equal(gb, gy.sum(0))


def test_frozen_linears_backpropagated_apart_and_after_an_in_place_change():
    from anima_trainer_sm120_b200 import fp8_quant
    g = torch.Generator(device=DEV).manual_seed(3)
    x = _randn(g, 256, 256).requires_grad_(True)
    W = _randn(g, 256, 256, std=0.05)
    Q, gy = fp8_quant.quantize_weight(W), _randn(g, 256, 256)
    y1, y2 = (fp8_quant.mxfp8_frozen_linear(x, Q, W) for _ in range(2))
    y1.backward(gy)
    first = x.grad.clone()
    y3 = fp8_quant.mxfp8_frozen_linear(x, Q, W)
    y2.backward(gy)
    y3.backward(gy)
    assert torch.equal(x.grad, (first + first) + first)
    h = x.detach().clone().requires_grad_(True) * 1.0
    a = fp8_quant.mxfp8_frozen_linear(h, Q, W)
    h.add_(1.0)
    b = fp8_quant.mxfp8_frozen_linear(h, Q, W)
    assert a.grad_fn is not b.grad_fn


def test_a_frozen_linear_belongs_to_the_graph_its_input_had_when_it_was_applied():
    """Same tensor object with another graph edge, and a bias computed from another linear of the same input."""
    from anima_trainer_sm120_b200 import fp8_quant
    g = torch.Generator(device=DEV).manual_seed(4)
    W = _randn(g, 256, 256, std=0.05)
    Q, gy = fp8_quant.quantize_weight(W), _randn(g, 256, 256)
    lin = lambda x, b=None: fp8_quant.mxfp8_frozen_linear(x, Q, W, b)
    base = _randn(g, 256, 256).requires_grad_(True)
    x = base * 1.0
    a = lin(x)
    x.detach_().requires_grad_(True)               # a leaf now; `a` still belongs to base's graph
    b = lin(x)
    assert a.grad_fn is not b.grad_fn
    ga, = torch.autograd.grad(a, base, gy)
    gb, = torch.autograd.grad(b, x, gy)
    assert torch.equal(ga, gb)
    y1 = lin(base)
    y2 = lin(base, y1.mean(0))                     # bias from the first output
    assert y1.grad_fn is not y2.grad_fn
    gx, = torch.autograd.grad(y2, base, gy)
    assert bool(torch.isfinite(gx).all())


def test_benchmark_step_runs_the_gemms_its_metric_counts():
    """The operands of bench.py: forward, input gradient and weight gradient, each seen by the GEMM timer and the launch
    counter. Without a gradient of x the same step has two GEMMs, so the count is of what ran."""
    import bench
    from anima_trainer_sm120_b200 import _lib, fp8_quant
    rows, bench_rows = 512, bench.M_ROWS
    try:
        bench.M_ROWS = rows
        s = bench.Shape(1024, 512, DEV, seed=0, host=False)
    finally:
        bench.M_ROWS = bench_rows
    lib, host = _lib.load(), _lib.host()
    for x, products in ((s.x, 3), (s.x.detach(), 2)):
        fp8_quant.clear_activation_memo()
        before = lib.anima_kernel_launches()
        host.time_gemms(True)
        fp8_quant.lokr_linear_fused(x, s.W, None, s.w1, s.w2, 1.0).backward(s.dy)
        host.time_gemms(False)
        times = host.gemm_times()
        assert [f for _, f in times] == [2.0 * rows * 1024 * 512] * products and all(ms > 0 for ms, _ in times)
        split = sum(lib.anima_mx_gemm_workspace_bytes(*mnk) > 0
                    for mnk in [(rows, 1024, 512), (1024, 512, rows), (rows, 512, 1024)][:products])
        # quantise x, merge, quantise dy, two Kronecker passes, the GEMMs and the finalize passes of split ones
        assert lib.anima_kernel_launches() - before == 5 + products + split
    assert s.x.grad is not None


def test_tensors_of_another_device_tangents_and_wrong_shapes_are_refused_before_a_launch():
    import torch.autograd.forward_ad as fwAD
    from anima_trainer_sm120_b200 import adaln_kernel, fp8_quant, tlokr
    from anima_trainer_sm120_b200.qk_norm_rope import FusedRMSNormRoPE
    g = torch.Generator(device=DEV).manual_seed(5)
    W, x = _randn(g, 256, 256, std=0.05), _randn(g, 64, 256)
    Q, bias = fp8_quant.quantize_weight(W), _randn(g, 256)
    w1, w2 = _randn(g, 8, 8), _randn(g, 32, 32)
    x5, mod = _randn(g, 1, 1, 4, 4, 256), _randn(g, 1, 1, 1, 1, 256)
    heads, w = _randn(g, 1, 16, 2, 128), _randn(g, 128)
    calls = [(lambda t: fp8_quant.mxfp8_frozen_linear(x, Q, W, t), bias),
             (lambda t: fp8_quant.lokr_linear_fused(x, W, t, w1, w2, 1.0), bias),
             (lambda t: fp8_quant.lokr_linear_fused(x, W, None, t, w2, 1.0), w1),
             (lambda t: adaln_kernel.fused_adaln(x5, t, mod, 1e-6), mod),
             (lambda t: adaln_kernel.fused_gated_add(x5, t, x5), mod),
             (lambda t: FusedRMSNormRoPE.apply(heads, t, None, None, 1e-6), w)]
    for call, t in calls:
        with pytest.raises(RuntimeError):
            call(t.cpu())
        with fwAD.dual_level(), pytest.raises(NotImplementedError):
            call(fwAD.make_dual(t, torch.ones_like(t)))
        call(t)
    big = fp8_quant.quantize_weight(_randn(g, 1024, 512, std=0.05))
    xt, a, b = _randn(g, 2, 128, 512), _randn(g, 128, 128), _randn(g, 128, 64)
    for args in [(w1, a, b, torch.ones(1, 128, device=DEV, dtype=BF16)), (w1, a, b, torch.ones(2, 64, device=DEV, dtype=BF16)),
                 (w1, a[:64], b, None), (w1, a, b[:64], None), (_randn(g, 4, 4), a, b, None)]:
        with pytest.raises((ValueError, NotImplementedError)):
            tlokr._MXTLoKrLinear.apply(xt, big, None, *args, 0.5)
    with pytest.raises(ValueError):
        adaln_kernel.fused_adaln(x5, mod, _randn(g, 1, 1, 1, 1, 128), 1e-6)
