"""What the native host path refuses before it looks for a device: its checks of shapes run first, so CPU tensors reach
them. A call that passes them is told that the kernels need CUDA tensors."""
from __future__ import annotations

import pytest
import torch

from anima_trainer_sm120_b200._lib import host

BF16 = torch.bfloat16
NONE = (None, None, None)


def _op(rows, k):
    """An operand as two tensors: codes and tiled scales."""
    return torch.zeros(rows, k, dtype=torch.uint8), torch.zeros(-(-rows // 128) * -(-k // 128) * 512, dtype=torch.uint8), None


def _bf16(*shape):
    return torch.zeros(*shape, dtype=BF16)


@pytest.mark.parametrize("rows,k,ok", [(64, 96, True), (128, 96, False), (32, 96, False), (64, 128, False), (96, 64, False)])
def test_backward_operand_of_a_frozen_linear_must_be_the_transpose_of_the_weight(rows, k, ok):
    x = _bf16(32, 64).requires_grad_(True)                  # weight [96, 64]: its column form is [64, 96]
    call = lambda t: host().frozen_linear(t, *_op(32, 64), *_op(96, 64), *_op(rows, k), None, None, False)
    with pytest.raises(RuntimeError if ok else ValueError, match="CUDA" if ok else "transpose"):
        call(x)
    with pytest.raises(RuntimeError, match="CUDA"):         # a pass without an input gradient does not read it
        call(x.detach())


def _tlinear(n, k, bias):
    col_ops = [t for op in (_op(n // 8, 128), _op(128, n // 8), _op(128, k // 8), _op(k // 8, 128)) for t in op[:2]]
    return host().tlinear(*_op(n, k)[:2], *_op(k, n)[:2], bias, _bf16(8, 8), _bf16(n // 8, 128), _bf16(128, k // 8), None, 1.0,
                          _bf16(8, 8), col_ops, False, True)


@pytest.mark.parametrize("which", ["lokr", "merged", "frozen", "mlp-1", "mlp-2", "tlokr", "tlokr-mlp-1", "tlokr-mlp-2"])
@pytest.mark.parametrize("short", [False, True])
def test_a_bias_that_is_not_one_value_per_output_is_refused(which, short):
    """The epilogue of the GEMM reads N values of it."""
    n, k = 512, 256
    cut = 32 if short else 0
    x, x_row, W = _bf16(64, k), _op(64, k), _bf16(n, k)
    b, b_in, b_out = _bf16(n - cut), (_bf16(n - cut if which.endswith("1") else n)), (_bf16(k - cut if which.endswith("2") else k))
    w1, w2, w2t = _bf16(8, 8), _bf16(n // 8, k // 8), _bf16(k // 8, n // 8)
    calls = {
        "lokr": lambda: host().lokr_linear(x, *x_row, *NONE, W, b, w1, w2, 1.0, False),
        "merged": lambda: host().merged_linear(x, *x_row, *NONE, W, b, False),
        "frozen": lambda: host().frozen_linear(x, *x_row, *_op(n, k), *NONE, None, b, False),
        "mlp": lambda: host().lokr_mlp(x, *x_row, *NONE, W, b_in, w1, w2, 1.0, _bf16(k, n), b_out, w1, w2t, 1.0, False),
        "tlokr": lambda: host().tlokr_linear(x, *x_row, _tlinear(n, k, b), False),
        "tlokr-mlp": lambda: host().tlokr_mlp(x, *x_row, _tlinear(n, k, b_in), _tlinear(k, n, b_out), False),
    }
    with pytest.raises(ValueError if short else RuntimeError, match="bias" if short else "CUDA"):
        calls[which[:-2] if which[-1] in "12" else which]()
