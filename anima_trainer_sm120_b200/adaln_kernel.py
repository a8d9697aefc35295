"""Fused AdaLN and gated-residual autograd ops with the call surface of
anima-trainer's ``adaln_kernel.py`` (``FusedAdaLN`` :157, ``fused_adaln`` :258,
``FusedGatedAdd`` :332, ``fused_gated_add`` :422), backed by the sm_100a kernels
in ``csrc/adaln.cu``.

Shapes follow the reference: ``x``/``y`` are ``(B, T, H, W, D)``, modulation
tensors are ``(B, T, 1, 1, D)`` and broadcast over ``(H, W)``. Statistics and all
elementwise math are fp32; results are stored in bf16. Unlike the reference the
``(H, W)`` reductions (dscale, dshift, dgate) are deterministic.
"""
from __future__ import annotations

import torch

from . import fp8_quant, ops
from ._lib import host

BF16 = torch.bfloat16

# When set, the AdaLN forward kernels also write the row-wise MXFP8 operand of their output (same pass, one
# more byte per element) and hand it to the quantised linears that consume the output through
# ``fp8_quant.adopt_row_operand``; those linears then launch no quantiser for it (the column-wise operand a
# trainable linear needs for its weight gradient is still made from y when asked for).
_EMIT_ROW_OPERAND = False


def emit_row_operand(enabled: bool = True) -> None:
    """Switch the quantise-in-the-producer forward on or off (off by default: it only pays when the consumers
    of the AdaLN output are this package's MXFP8 linears)."""
    global _EMIT_ROW_OPERAND
    _EMIT_ROW_OPERAND = bool(enabled)


def _emits(x: torch.Tensor, rows: int, d: int) -> bool:
    return _EMIT_ROW_OPERAND and x.dtype == BF16 and ops.can_emit_row_codes(rows, d)


def _adopt(y: torch.Tensor, made: tuple) -> None:
    """Hand the row-wise operand the kernel wrote (if it did) to the linears that consume y."""
    op = ops.operand(made)
    if op is not None:
        fp8_quant.adopt_row_operand(y, op)


def _rows_of(x: torch.Tensor, mod: torch.Tensor) -> tuple[int, int]:
    """(rows, D) of an activation; the modulation tensor must have one row per (batch, time)."""
    B, T, H, W, D = x.shape
    N, M = B * T * H * W, mod.numel() // D if D else 0
    assert N == M * H * W, f"shape mismatch: N={N}, M={M}, HW={H * W}"
    return N, D


def _need_bf16_stream(name: str, *tensors: torch.Tensor) -> None:
    """The kernels store bf16. The reference's ops keep the input dtype (``torch.empty_like(x_flat)``,
    adaln_kernel.py:185-187), so an fp32 residual stream would be rounded to bf16 at every sublayer here without
    notice; it is refused instead (modulation tensors of another dtype are cast, their gradients cast back)."""
    for t in tensors:
        if t.dtype != BF16:
            raise TypeError(f"{name}: activations must be bfloat16, got {t.dtype} (the fused kernels have no "
                            "fp32-stream form; use the block's unpatched forward for use_fp32)")


class FusedAdaLN:
    """``LayerNorm(x, no affine, eps) * (1 + scale) + shift`` (native node: ``csrc/host/norm.cpp``)."""

    @staticmethod
    def apply(x, scale, shift, eps):
        assert x.is_cuda, "FusedAdaLN requires CUDA tensors"
        _need_bf16_stream("FusedAdaLN", x)
        N, D = _rows_of(x, scale)
        y, made = host().adaln(x, scale, shift, eps, _emits(x, N, D))
        _adopt(y, made)
        return y


def fused_adaln(x: torch.Tensor, scale: torch.Tensor, shift: torch.Tensor, eps: float) -> torch.Tensor:
    return FusedAdaLN.apply(x, scale, shift, eps)


class FusedGatedAdd:
    """``out = x + gate * y``; backward ``dx = dout``, ``dy = gate * dout``,
    ``dgate = sum_{h,w}(dout * y)``."""

    @staticmethod
    def apply(x, gate, y):
        assert x.is_cuda, "FusedGatedAdd requires CUDA tensors"
        assert x.shape == y.shape, f"x {x.shape} != y {y.shape}"
        _need_bf16_stream("FusedGatedAdd", x, y)
        _rows_of(x, gate)
        return host().gated_add(x, gate, y)


def fused_gated_add(x: torch.Tensor, gate: torch.Tensor, y: torch.Tensor) -> torch.Tensor:
    return FusedGatedAdd.apply(x, gate, y)


class FusedGatedAddAdaLN:
    """``x_new = x + gate * sub`` followed by ``y = AdaLN(x_new; scale, shift)``: the residual update of one
    sublayer and the modulation of the next, from one read of x and sub. Returns ``(x_new, y)``, each
    bit-identical to ``FusedGatedAdd`` then ``FusedAdaLN``; backward is one kernel too (the AdaLN input
    gradient, its sum with the residual-stream gradient, and the gated-residual backward), again bit-identical
    to the separate kernels."""

    @staticmethod
    def apply(x, gate, sub, scale, shift, eps):
        assert x.is_cuda, "FusedGatedAddAdaLN requires CUDA tensors"
        assert x.shape == sub.shape, f"x {x.shape} != sub {sub.shape}"
        _need_bf16_stream("FusedGatedAddAdaLN", x, sub)
        N, D = _rows_of(x, gate)
        _rows_of(x, scale)
        x_new, y, made = host().gated_add_adaln(x, gate, sub, scale, shift, eps, _emits(x, N, D))
        _adopt(y, made)
        return x_new, y


def fused_gated_add_adaln(x, gate, sub, scale, shift, eps):
    return FusedGatedAddAdaLN.apply(x, gate, sub, scale, shift, eps)
