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
    call = lambda t: host().frozen_linear(t, *_op(32, 64), *_op(96, 64), *_op(rows, k), None, None)
    with pytest.raises(RuntimeError if ok else ValueError, match="CUDA" if ok else "transpose"):
        call(x)
    with pytest.raises(RuntimeError, match="CUDA"):         # a pass without an input gradient does not read it
        call(x.detach())
