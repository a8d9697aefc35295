"""Timestep-aware LoKr (T-LoKr) with the call surface of anima-trainer's ``tlokr.py``.

``W2`` of a full-matrix LoKr adapter is factored as ``A @ B`` (rank r) and a per-sample prefix
of that rank is active: ``active(t) = floor((r - r_min) * (1 - t) + r_min)`` (reference
``active_rank_for_timestep`` :40-57, mask :84-92). The adapter output for a linear input is
evaluated structurally (reference :472-492), never forming ``kron(W1, A @ B)``:

    grouped = x.view(B, L*, uq, vq);  hidden = grouped @ B.T;  mixed = W1 @ (hidden * mask)
    out = mixed @ A.T  ->  (B, L*, up * vp)

Mirrored interface: ``active_rank_for_timestep``, ``set_timestep`` / ``clear_timestep`` (:110-130),
``install_root_timestep_hooks`` (:270-292), ``convert_network`` (:330-448), ``_StructuredLoKr``
(:451-540), ``_FP8StructuredLoKr`` (:543-676, here MXFP8), ``forward`` (:738-759).

Kernels: the 8x8 mix, its transpose and its fp32 weight gradient run in ``csrc/tlokr_mix.cu``;
in the quantised variant the factor GEMMs (2 forward, 2 recomputed + 4 in backward) run as
MXFP8 tcgen05 GEMMs with the quantiser producing both operand forms per tensor. The bf16
variant uses ``torch.matmul`` for the factor GEMMs (a library GEMM, as in the reference).
"""
from __future__ import annotations

import math
import os
from contextvars import ContextVar
from dataclasses import dataclass, field
from types import MethodType

from typing import NamedTuple

import torch
import torch.nn as nn
import torch.nn.functional as F

from . import ops
from ._lib import host
from .tlokr_kernels import rank_mix, rank_mix_wgrad

_FORMAT_VERSION = 1
BF16 = torch.bfloat16


def active_rank_for_timestep(timestep: float, *, max_rank: int, min_rank: int) -> int:
    """Prefix rank for a scalar flow timestep (t = 1 is the noisiest point)."""
    if max_rank <= 0:
        raise ValueError(f"max_rank must be positive; got {max_rank}")
    if not 1 <= min_rank <= max_rank:
        raise ValueError(f"min_rank must be in [1, {max_rank}]; got {min_rank}")
    t = min(1.0, max(0.0, float(timestep)))
    return max(min_rank, min(max_rank, math.floor((max_rank - min_rank) * (1.0 - t) + min_rank)))


@dataclass
class _TimestepState:
    timesteps: torch.Tensor
    uniform_timestep: float | None = None   # known single timestep: factors are sliced, no mask
    masks: dict = field(default_factory=dict)

    def mask(self, *, max_rank: int, min_rank: int, dtype: torch.dtype, device: torch.device) -> torch.Tensor:
        """[B, max_rank] 0/1 prefix mask; built once per forward and shared by all modules."""
        key = (max_rank, min_rank, dtype, device)
        hit = self.masks.get(key)
        if hit is None:
            t = self.timesteps.detach().to(device=device, dtype=torch.float32).reshape(-1)
            active = torch.floor((max_rank - min_rank) * (1.0 - t.clamp(0.0, 1.0)) + min_rank).to(torch.int64)
            active.clamp_(min=min_rank, max=max_rank)
            hit = (torch.arange(max_rank, device=device).unsqueeze(0) < active.unsqueeze(1)).to(dtype)
            self.masks[key] = hit
        return hit


_STATE: ContextVar[_TimestepState | None] = ContextVar("anima_b200_tlokr_state", default=None)


def set_timestep(timesteps: torch.Tensor, *, uniform_timestep: float | None = None) -> None:
    """Set the timestep context for every T-LoKr module; it stays live through backward because
    activation checkpointing re-runs adapter forwards there. Pair with :func:`clear_timestep`."""
    if not torch.is_tensor(timesteps):
        raise TypeError("T-LoKr timesteps must be a torch.Tensor")
    _STATE.set(_TimestepState(timesteps=timesteps, uniform_timestep=uniform_timestep))


def clear_timestep() -> None:
    _STATE.set(None)


def _current_state() -> _TimestepState:
    state = _STATE.get()
    if state is None:
        raise RuntimeError("T-LoKr forward has no timestep context; call "
                           "anima_trainer_sm120_b200.tlokr.set_timestep() around the DiT forward")
    return state


def install_root_timestep_hooks(dit: nn.Module) -> None:
    """Derive a context from the root forward's ``timesteps`` argument when none was set explicitly,
    restore the previous one afterwards, and keep it alive for checkpoint recomputation: each
    block's ``_forward`` is wrapped so the callable the checkpoint retains re-enters the state."""
    if getattr(dit, "_tlokr_timestep_hooks_installed", False):
        return

    def pre(_m, args, kwargs):
        if _STATE.get() is not None:
            dit._tlokr_tokens.append(None)
            return
        t = next((kwargs[k] for k in ("timesteps", "timesteps_B_T", "timestep") if kwargs.get(k) is not None), None)
        if t is None and len(args) >= 2:
            t = args[1]
        if not torch.is_tensor(t):
            raise RuntimeError("T-LoKr could not derive a tensor timestep from the DiT forward arguments")
        dit._tlokr_tokens.append(_STATE.set(_TimestepState(timesteps=t)))

    def post(_m, _args, _kwargs, _out):
        token = dit._tlokr_tokens.pop() if dit._tlokr_tokens else None
        if token is not None:
            _STATE.reset(token)

    dit._tlokr_tokens = []
    dit.register_forward_pre_hook(pre, with_kwargs=True)
    dit.register_forward_hook(post, with_kwargs=True, always_call=True)
    for blk in dit.modules():
        if hasattr(blk, "_forward") and hasattr(blk, "gradient_checkpointing") and "_forward" not in blk.__dict__:

            def contextual(self_blk, *a, **kw):
                # the class attribute is looked up at call time so that a later adaln_patch.install() is honoured
                inner = type(self_blk)._forward
                captured = getattr(self_blk, "_tlokr_captured_state", None)
                if _STATE.get() is not None or captured is None:
                    self_blk._tlokr_captured_state = _STATE.get()
                    return inner(self_blk, *a, **kw)
                token = _STATE.set(captured)        # recomputation during backward, on autograd's thread
                try:
                    return inner(self_blk, *a, **kw)
                finally:
                    _STATE.reset(token)

            object.__setattr__(blk, "_forward", MethodType(contextual, blk))
    dit._tlokr_timestep_hooks_installed = True


def convert_network(network: nn.Module, *, rank: int, min_rank_ratio: float) -> int:
    """Convert freshly created full-matrix LoKr adapters in place: ``lokr_w2`` becomes the pair
    ``lokr_w2_a`` (kaiming-uniform) / ``lokr_w2_b`` (zeros), so the adapted model starts at the base
    model exactly. Returns the number of converted modules."""
    from .lokr import LokrModule

    if rank <= 0:
        raise ValueError(f"T-LoKr rank must be positive; got {rank}")
    if not 0.0 < min_rank_ratio <= 1.0:
        raise ValueError(f"T-LoKr min_rank_ratio must be in (0, 1]; got {min_rank_ratio}")
    min_rank = max(1, min(rank, math.ceil(rank * min_rank_ratio)))
    pending = list(getattr(network, "unet_loras", ()))
    converted = 0
    for module in (pending if pending else list(network.modules())):
        if not isinstance(module, LokrModule):
            continue
        if module.module_type != "linear":
            raise TypeError(f"T-LoKr supports Linear targets only; {module.lora_name} wraps {module.module_type}")
        if not module.use_w1 or not module.use_w2:
            raise ValueError(f"{module.lora_name}: T-LoKr conversion requires full_matrix=true")
        if module.wd or module.bypass_mode:
            raise ValueError(f"{module.lora_name}: T-LoKr does not support weight decomposition or bypass mode")
        if module.rank_dropout or module.dropout:
            raise ValueError(f"{module.lora_name}: T-LoKr does not support rank/dropout")
        old = module.lokr_w2
        vp, vq = old.shape
        if rank > min(vp, vq):
            raise ValueError(f"T-LoKr rank {rank} exceeds the large Kronecker factor {tuple(old.shape)} "
                             f"in {module.lora_name}")
        del module.lokr_w2
        a = nn.Parameter(torch.empty(vp, rank, device=old.device, dtype=old.dtype))
        b = nn.Parameter(torch.zeros(rank, vq, device=old.device, dtype=old.dtype))
        nn.init.kaiming_uniform_(a, a=math.sqrt(5))
        module.register_parameter("lokr_w2_a", a)
        module.register_parameter("lokr_w2_b", b)
        module.use_w2 = False
        module.full_matrix = False
        module.lora_dim = rank
        module._tlokr_enabled, module._tlokr_rank, module._tlokr_min_rank = True, rank, min_rank
        scalar = module.scalar.item() if torch.is_tensor(module.scalar) else module.scalar
        module._tlokr_alpha = float(module.scale) * float(scalar) * float(module.multiplier)
        module.register_buffer("tlokr_schedule", torch.tensor([_FORMAT_VERSION, rank, min_rank], dtype=torch.int32))
        converted += 1
    if converted == 0:
        raise RuntimeError("T-LoKr conversion found no LoKr modules")
    network._tlokr_enabled, network._tlokr_rank, network._tlokr_min_rank = True, rank, min_rank
    return converted


def _grouped(x: torch.Tensor, uq: int) -> torch.Tensor:
    return x.reshape(x.shape[0], -1, uq, x.shape[-1] // uq)


class _StructuredLoKr(torch.autograd.Function):
    """bf16 structured delta with manual backward; saves only x and the small factors and
    recomputes the rank-space intermediates per module in backward (reference :451-540)."""

    @staticmethod
    def forward(ctx, x, w1, w2_a, w2_b, mask):
        dt = x.dtype
        c, a, b = w1.to(dt), w2_a.to(dt), w2_b.to(dt)
        hidden = torch.matmul(_grouped(x, c.shape[1]), b.t())
        out = torch.matmul(rank_mix(hidden, c, mask), a.t())
        ctx.save_for_backward(x, w1, w2_a, w2_b, *(() if mask is None else (mask,)))
        ctx.has_mask = mask is not None
        return out.reshape(*x.shape[:-1], -1)

    @staticmethod
    def backward(ctx, grad_output):
        saved = ctx.saved_tensors        # read once: activation checkpointing unpacks on access
        x, w1, w2_a, w2_b = saved[:4]
        mask = saved[4] if ctx.has_mask else None
        dt = x.dtype
        c, a, b = w1.to(dt), w2_a.to(dt), w2_b.to(dt)
        up, uq = c.shape
        vp = a.shape[0]
        grouped = _grouped(x, uq)
        hidden = torch.matmul(grouped, b.t())
        mixed = rank_mix(hidden, c, mask)
        g_blocks = grad_output.to(dt).reshape(x.shape[0], -1, up, vp)
        g_a = g_blocks.reshape(-1, vp).t() @ mixed.reshape(-1, mixed.shape[-1])
        g_mixed = torch.matmul(g_blocks, a)
        g_c = rank_mix_wgrad(g_mixed, hidden, mask)
        g_hidden = rank_mix(g_mixed, c, mask, transpose=True)
        g_b = g_hidden.reshape(-1, g_hidden.shape[-1]).t() @ grouped.reshape(-1, grouped.shape[-1])
        g_x = torch.matmul(g_hidden, b).reshape(x.shape)
        return g_x.to(x.dtype), g_c.to(w1.dtype), g_a.to(w2_a.dtype), g_b.to(w2_b.dtype), None


def _capturing(p: torch.Tensor) -> bool:
    """Inside a CUDA-graph capture the factor conversions must be recorded with the rest of the step: a form kept
    from an earlier call would be baked into the graph and every replay would multiply by the factors of the step
    that was captured."""
    return p.is_cuda and torch.cuda.is_current_stream_capturing()


def _factor_forms(p: torch.Tensor, *, quantise: bool):
    """bf16 copy (``quantise=False``) or both MXFP8 operands (``quantise=True``) of a small adapter factor.

    A checkpointed step reads every factor three times with the same values (first pass, recomputation,
    backward); for a leaf parameter the result is kept on the parameter object, keyed on its in-place version
    counter and storage address (an optimizer step or a reassigned ``.data`` invalidates it), which removes two
    thirds of these tiny launches. Sliced or computed factors are converted on every call."""
    cacheable = p.is_leaf and isinstance(p, nn.Parameter) and not _capturing(p)
    slot = "_anima_mx_forms" if quantise else "_anima_bf16_form"
    key = (p._version, p.data_ptr())
    if cacheable:
        hit = getattr(p, slot, None)
        if hit is not None and hit[0] == key:
            return hit[1]
    with torch.no_grad():
        val = _q(p.detach(), col=True) if quantise else p.detach().to(BF16).contiguous()
    if cacheable:
        setattr(p, slot, (key, val))
    return val


def _scaled_row_form(p: torch.Tensor, alpha: float) -> ops.MXOperand:
    """Row-wise MXFP8 operand of ``alpha * p`` rounded to bf16 (the factor a folded delta multiplies by), kept on
    a leaf parameter like :func:`_factor_forms`."""
    cacheable = p.is_leaf and isinstance(p, nn.Parameter) and not _capturing(p)
    key = (p._version, p.data_ptr(), float(alpha))
    if cacheable:
        hit = getattr(p, "_anima_mx_scaled_row", None)
        if hit is not None and hit[0] == key:
            return hit[1]
    with torch.no_grad():
        val = ops.mx_quantize((p.detach().float() * float(alpha)).to(BF16).contiguous(), rowwise=True)[0]
    if cacheable:
        p._anima_mx_scaled_row = (key, val)
    return val


# Fold the structured delta into the base GEMMs as extra K-blocks (``ops.mx_gemm_delta``) where the shapes allow:
# the base projection and ``+ alpha * delta`` (forward), the base input gradient and ``+ grad_hidden @ B``
# (backward) are then one GEMM each, and the output is neither re-read nor rounded twice. False keeps the
# separate add-GEMMs (for comparison; ANIMA_TLOKR_FOLD_DELTA=0 sets it at import).
FOLD_DELTA = os.environ.get("ANIMA_TLOKR_FOLD_DELTA", "1") != "0"


# Compute hidden, the mix and the quantisation of the mixed tensor in one kernel in the forward chain
# (``ops.tlokr_hidden_mix_planes``); False runs the factor GEMM and the quantising mix as two kernels (same bits).
FUSE_HIDDEN_MIX = os.environ.get("ANIMA_TLOKR_FUSE_HIDDEN_MIX", "1") != "0"


def _q(t2d: torch.Tensor, *, col: bool = False):
    return ops.mx_quantize(t2d.contiguous() if t2d.dtype == BF16 else t2d.to(BF16).contiguous(),
                           rowwise=True, colwise=col)


class _MXStructuredLoKr(torch.autograd.Function):
    """The same delta with every factor GEMM in MXFP8 on the tensor cores (the reference's
    ``_FP8StructuredLoKr`` uses TE block-FP8 for them); the 8x8 mix stays in bf16.

    With ``base`` given the result is ``base + alpha * delta``, formed in the epilogue of the last GEMM
    (the reference's separate ``torch.add(base, delta, alpha=)``, ``tlokr.py:757-759``)."""

    @staticmethod
    def forward(ctx, x, w1, w2_a, w2_b, mask, base=None, alpha: float = 1.0):
        c = w1.to(BF16)
        aq, aq_col = _q(w2_a.detach(), col=True)      # A [vp, r]: row form for out, column form for dgrad
        bq, bq_col = _q(w2_b.detach(), col=True)      # B [r, vq]
        grouped = _grouped(x, c.shape[1])
        g2 = grouped.reshape(-1, grouped.shape[-1])
        gq, _ = _q(g2)
        hidden = ops.mx_gemm(gq, bq).view(*grouped.shape[:-1], w2_b.shape[0])
        mixed = rank_mix(hidden, c, mask)
        mq, _ = _q(mixed.reshape(-1, mixed.shape[-1]))
        ctx.save_for_backward(x, w1, w2_a, w2_b, *(() if mask is None else (mask,)))
        ctx.has_mask, ctx.ops = mask is not None, (aq_col, bq, bq_col)
        ctx.has_base, ctx.alpha = base is not None, float(alpha) if base is not None else 1.0
        if base is None:
            return ops.mx_gemm(mq, aq).view(*x.shape[:-1], -1).to(x.dtype)
        # base (bf16, contiguous) is updated in place: base += alpha * delta, added by the GEMM's stores
        res = base.view(-1, w2_a.shape[0])
        ops.mx_gemm(mq, aq, residual=res, alpha=float(alpha), out=res)
        ctx.mark_dirty(base)
        return base

    @staticmethod
    def backward(ctx, grad_output):
        saved = ctx.saved_tensors        # read once: activation checkpointing unpacks on access
        x, w1, w2_a, w2_b = saved[:4]
        mask = saved[4] if ctx.has_mask else None
        aq_col, bq, bq_col = ctx.ops
        c = w1.to(BF16)
        up, uq = c.shape
        vp, rank = w2_a.shape
        grouped = _grouped(x, uq)
        g2 = grouped.reshape(-1, grouped.shape[-1])
        gq, gq_col = _q(g2, col=True)
        hidden = ops.mx_gemm(gq, bq).view(*grouped.shape[:-1], rank)
        mixed = rank_mix(hidden, c, mask)
        _, mq_col = _q(mixed.reshape(-1, rank), col=True)
        gb2 = grad_output.reshape(-1, vp)
        gbq, gbq_col = _q(gb2, col=True)
        g_a = ops.mx_gemm(gbq_col, mq_col, out_dtype=torch.float32, alpha=ctx.alpha)   # alpha * grad_blocks^T @ mixed [vp, r]
        g_mixed = ops.mx_gemm(gbq, aq_col, alpha=ctx.alpha).view(*mixed.shape)         # alpha * grad_blocks @ A       [.., r]
        g_c = rank_mix_wgrad(g_mixed, hidden, mask)
        g_hidden = rank_mix(g_mixed, c, mask, transpose=True)
        ghq, ghq_col = _q(g_hidden.reshape(-1, rank), col=True)
        g_b = ops.mx_gemm(ghq_col, gq_col, out_dtype=torch.float32)          # grad_hidden^T @ grouped [r, vq]
        g_x = ops.mx_gemm(ghq, bq_col).view(x.shape)                         # grad_hidden @ B
        return (g_x.to(x.dtype), g_c.to(w1.dtype), g_a.to(w2_a.dtype), g_b.to(w2_b.dtype), None,
                grad_output if ctx.has_base else None, None)


_FP8StructuredLoKr = _MXStructuredLoKr  # name used by anima-trainer


def _delta_plan(module, x: torch.Tensor, *, fp8: bool):
    """(autograd function, A, B, mask) of the structured delta for the current timestep context
    (the dispatch of reference :679-735)."""
    state = _current_state()
    rank, min_rank = module._tlokr_rank, module._tlokr_min_rank
    w1 = module.lokr_w1
    if x.shape[-1] % w1.shape[1]:
        raise RuntimeError(f"{module.lora_name}: input width {x.shape[-1]} is not divisible by the W1 "
                           f"input factor {w1.shape[1]}")
    if state.uniform_timestep is not None:
        # One known timestep for the whole batch: slice the factors to the active prefix, which drops the
        # mask and the inactive-rank work. The mix kernel wants the rank in multiples of 8 (the MXFP8 GEMMs in
        # multiples of 32); other prefixes keep the full factors and use an equivalent uniform mask.
        active = active_rank_for_timestep(state.uniform_timestep, max_rank=rank, min_rank=min_rank)
        if active % 8 == 0:
            fn = _MXStructuredLoKr if fp8 and active % 32 == 0 else _StructuredLoKr
            return fn, module.lokr_w2_a[:, :active], module.lokr_w2_b[:active], None
        key = ("uniform", rank, active, x.dtype, x.device, x.shape[0])
        mask = state.masks.get(key)
        if mask is None:
            mask = (torch.arange(rank, device=x.device) < active).to(x.dtype).expand(x.shape[0], rank).contiguous()
            state.masks[key] = mask
        return (_MXStructuredLoKr if fp8 else _StructuredLoKr), module.lokr_w2_a, module.lokr_w2_b, mask
    mask = state.mask(max_rank=rank, min_rank=min_rank, dtype=x.dtype, device=x.device)
    if x.shape[0] != mask.shape[0]:
        raise RuntimeError(f"{module.lora_name}: activation batch {x.shape[0]} does not match timestep "
                           f"batch {mask.shape[0]}")
    return (_MXStructuredLoKr if fp8 else _StructuredLoKr), module.lokr_w2_a, module.lokr_w2_b, mask


def _structured_delta(module, x: torch.Tensor, *, fp8: bool, base: torch.Tensor | None = None,
                      alpha: float = 1.0) -> torch.Tensor:
    """``x @ kron(W1, A @ B).T`` for the current timestep context; with ``base`` given,
    ``base + alpha * delta`` (fused into the last GEMM on the quantised path)."""
    fn, w2_a, w2_b, mask = _delta_plan(module, x, fp8=fp8)
    args = (x, module.lokr_w1, w2_a, w2_b, mask)
    if base is None:
        return fn.apply(*args)
    if fn is _MXStructuredLoKr and base.dtype == BF16 and base.is_contiguous() and base.requires_grad:
        return fn.apply(*args, base, alpha)
    return torch.add(base, fn.apply(*args), alpha=alpha)


def _tlinear(W_mx, bias, w1, w2_a, w2_b, mask, alpha: float):
    """The native description of one quantised T-LoKr linear: base operands, parameters, mask and the factors'
    forms (kept per parameter version by :func:`_factor_forms`)."""
    c = _factor_forms(w1, quantise=False)
    forms = []
    for p in (w2_a, w2_b):                               # A [vp, r], B [r, vq]: row and column operands of each
        for op in _factor_forms(p, quantise=True):
            forms += (op.codes, op.scales)
    if FOLD_DELTA and w2_a.shape[1] == 128:              # alpha * A, the factor a folded delta multiplies by
        op = _scaled_row_form(w2_a, alpha)
        forms += (op.codes, op.scales)
    col = (None, None) if W_mx.col is None else (W_mx.col.codes, W_mx.col.scales)
    return host().tlinear(W_mx.row.codes, W_mx.row.scales, *col, bias, w1, w2_a, w2_b, mask, float(alpha), c, forms,
                          FOLD_DELTA, FUSE_HIDDEN_MIX)


def _row_operand_unless_kept(x, *trainable):
    """Row-wise operand of x for a pass that backward will not read, else nothing: the node then quantises the
    grouped view of x in both forms itself, and its row codes serve the base GEMM too."""
    from .fp8_quant import _native, _wants_grad, in_first_pass, quantize_activation
    first = in_first_pass()
    if _wants_grad(x, *trainable) and not first:
        return (None, None, None), first
    return _native(quantize_activation(x, colwise=False)[0]), first


class _MXTLoKrLinear:
    """The whole quantised T-LoKr linear, ``x W^T + bias + alpha * delta(x)``, as ONE autograd node
    (native: ``csrc/host/tlokr.cpp``).

    The reference runs a frozen FP8 base projection (``fp8_frozen_linear``, ``tlokr.py:743``), the
    structured delta (``_FP8StructuredLoKr``, :543-676) and ``torch.add(base, delta, alpha=)`` (:757-759) as
    three nodes, each quantising its own inputs. As one node x and the incoming gradient are quantised once each,
    and the delta enters the base GEMMs (forward and input gradient) as extra K-blocks where the shape allows."""

    @staticmethod
    def apply(x, W_mx, bias, w1, w2_a, w2_b, mask, alpha: float):
        x_row, first = _row_operand_unless_kept(x, w1, w2_a, w2_b, bias)
        return host().tlokr_linear(x, *x_row, _tlinear(W_mx, bias, w1, w2_a, w2_b, mask, alpha), first)


class _MXTLoKrMLP:
    """``layer2(gelu(layer1(x)))`` with both layers quantised T-LoKr linears, as one native node: the activation and
    its derivative are evaluated inside the quantiser, so neither ``gelu(h)`` nor ``grad * gelu'(h)`` is ever written
    as a bf16 tensor."""

    @staticmethod
    def apply(x, W1, b1, w1_1, a_1, b_1, mask1, alpha1: float, W2, b2, w1_2, a_2, b_2, mask2, alpha2: float):
        x_row, first = _row_operand_unless_kept(x, w1_1, a_1, b_1, w1_2, a_2, b_2)
        return host().tlokr_mlp(x, *x_row, _tlinear(W1, b1, w1_1, a_1, b_1, mask1, alpha1),
                                _tlinear(W2, b2, w1_2, a_2, b_2, mask2, alpha2), first)


class _ActSpec(NamedTuple):
    """Shape, dtype and device of an activation: all the dispatch looks at."""
    shape: tuple
    dtype: torch.dtype
    device: torch.device


def single_node_plan(module, x):
    """Arguments ``(W_mx, bias, w1, A, B, mask, alpha)`` of the one-node quantised T-LoKr linear for an input
    ``x`` (a tensor or an :class:`_ActSpec`), or None when the call has to take the general path (no
    pre-quantised base, rows not a multiple of 32, input not bf16 on CUDA, a factor other than 8 x 8, or an active
    rank the MXFP8 GEMMs cannot contract)."""
    base_q = getattr(module, "_tlokr_fp8_base_weight", None)
    rows = 1
    for d in x.shape[:-1]:
        rows *= d
    if (base_q is None or base_q.col is None or x.device.type != "cuda" or x.dtype != BF16
            or rows % 32 or tuple(module.lokr_w1.shape) != (8, 8)):
        return None
    fn, w2_a, w2_b, mask = _delta_plan(module, x, fp8=True)
    if fn is not _MXStructuredLoKr:
        return None
    return base_q, module.org_module[0].bias, module.lokr_w1, w2_a, w2_b, mask, module._tlokr_alpha


# Precision of the structured delta when the base projection is quantised: "mxfp8" (every factor GEMM on the
# MXFP8 tensor path, the reference's FP8 mode) or "bf16" (the HBM-bound factor chain stays in bf16 and skips its
# quantisation passes; the base projection stays MXFP8).
DELTA_PRECISION = "mxfp8"


def forward(module, x: torch.Tensor) -> torch.Tensor:
    """T-LoKr forward called by ``lokr_patch``: frozen base projection (quantised once when
    ``fp8_quant.quantize_tlokr_base_weights`` ran) plus ``alpha`` times the structured delta."""
    org = module.org_module[0]
    base_q = getattr(module, "_tlokr_fp8_base_weight", None)
    quantised = base_q is not None and x.is_cuda and (x.numel() // x.shape[-1]) % 32 == 0
    plan = single_node_plan(module, x) if DELTA_PRECISION == "mxfp8" else None
    if plan is not None:
        return _MXTLoKrLinear.apply(x.contiguous(), *plan)
    if quantised:
        from .fp8_quant import fp8_frozen_linear
        base = fp8_frozen_linear(x, base_q, org.weight, org.bias)
    else:
        base = F.linear(x, org.weight, org.bias)
    return _structured_delta(module, x, fp8=quantised and DELTA_PRECISION == "mxfp8", base=base,
                             alpha=module._tlokr_alpha)
