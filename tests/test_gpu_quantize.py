"""GPU parity: the MXFP8 quantiser through the C ABI vs the CPU oracle — bit-exact codes and
scale bytes — on the golden vectors, on seeded data with config-2 statistics, on ragged and
edge shapes, and at full size through size-independent properties."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import bf16_from_bits
from oracle import mxfp8 as OQ

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True, params=["1", "2"], ids=["plain-loads", "copy-engine-fed"])
def quantiser_variant(request, monkeypatch):
    """Every test of this module runs once per quantiser kernel (the library reads the variable on every call):
    the tile kernel with plain loads, and the persistent kernel fed by bulk tensor copies."""
    monkeypatch.setenv("ANIMA_MX_QUANTIZE_VARIANT", request.param)
    yield request.param
    from anima_trainer_sm120_b200 import _lib
    assert _lib.load().anima_mx_quantize_status() == 0


def _ops():
    from anima_trainer_sm120_b200 import ops
    return ops


def _activations(rows, cols, seed, outliers=True):
    """bf16 ~N(0,1) with 0.1 % of the channels scaled x50 (config 2)."""
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(rows, cols, generator=g)
    if outliers:
        idx = torch.randperm(cols, generator=g)[: max(1, -(-cols // 1000))]
        x[:, idx] *= 50.0
    return x.to(torch.bfloat16)


def _check(x_cpu, *, rowwise, colwise, layout):
    ops = _ops()
    xf = x_cpu.float().numpy()
    row, col = ops.mx_quantize(x_cpu.cuda(), rowwise=rowwise, colwise=colwise, layout=layout)
    torch.cuda.synchronize()
    if rowwise:
        codes, scales = OQ.quantize_rowwise(xf)
        assert np.array_equal(row.codes.cpu().numpy(), codes)
        want = scales if layout == 0 else OQ.scales_to_tiled(scales)
        assert np.array_equal(row.scales.cpu().numpy().reshape(want.shape), want)
    if colwise:
        codes, scales = OQ.quantize_colwise_T(xf)
        assert np.array_equal(col.codes.cpu().numpy(), codes)
        want = scales if layout == 0 else OQ.scales_to_tiled(scales)
        assert np.array_equal(col.scales.cpu().numpy().reshape(want.shape), want)


def test_golden_vectors_bit_exact(golden):
    """Scale bytes equal the reference quantiser's everywhere; codes equal the oracle's, which the
    golden test pins against the reference (hardware round-to-nearest-even cast)."""
    ops = _ops()
    g = golden("quantiser")
    x = bf16_from_bits(g["x"])
    row, col = ops.mx_quantize(x.cuda(), rowwise=True, colwise=True, layout=0)
    assert np.array_equal(row.scales.cpu().numpy(), g["scales"])
    codes, _ = OQ.quantize_rowwise(x.float().numpy())
    assert np.array_equal(row.codes.cpu().numpy(), codes)
    w = bf16_from_bits(g["w"])
    _, wcol = ops.mx_quantize(w.cuda(), rowwise=False, colwise=True, layout=0)
    assert np.array_equal(wcol.scales.cpu().numpy(), g["dgrad_scales"])
    # dequantise of the reference's codes reproduces the reference's dequantize_rowwise bits
    op = ops.MXOperand(torch.from_numpy(g["codes"]).cuda(), torch.from_numpy(g["scales"]).cuda(), 0)
    deq = ops.mx_dequantize(op).cpu()
    assert torch.equal(deq.view(torch.int16), bf16_from_bits(g["deq"]).view(torch.int16))


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("rows,cols", [(128, 128), (256, 384), (32, 32), (96, 160), (160, 2048), (512, 96)])
def test_row_and_column_forms_bit_exact(rows, cols, layout):
    _check(_activations(rows, cols, seed=rows * 7 + cols), rowwise=True, colwise=True, layout=layout)


@pytest.mark.parametrize("layout", [0, 1])
def test_ragged_rows_rowwise_only(layout):
    # rows not a multiple of 32 (row-wise form only needs cols % 32 == 0), incl. a single row
    for rows, cols in [(1, 64), (45, 96), (130, 256)]:
        _check(_activations(rows, cols, seed=rows), rowwise=True, colwise=False, layout=layout)


def test_column_only_and_strided_input():
    _check(_activations(64, 200, seed=3), rowwise=False, colwise=True, layout=1)
    ops = _ops()
    big = _activations(64, 512, seed=9).cuda()
    view = big[:, 128:384]                       # row pitch 512, 256 columns
    row, _ = ops.mx_quantize(view, rowwise=True, layout=0)
    codes, scales = OQ.quantize_rowwise(view.cpu().float().numpy())
    assert np.array_equal(row.codes.cpu().numpy(), codes) and np.array_equal(row.scales.cpu().numpy(), scales)


def test_edge_values():
    x = torch.zeros(32, 64, dtype=torch.bfloat16)
    x[0, :] = 0.0
    x[1, :32] = float("inf"); x[1, 32:] = -3.0e38
    x[2, :] = 1e-38
    x[3, 0] = 448.0; x[3, 1] = -449.0; x[3, 2] = 1.75
    x[4, :] = torch.tensor(2.0 ** -126)
    _check(x, rowwise=True, colwise=True, layout=0)


def test_empty_input_is_a_noop():
    ops = _ops()
    row, _ = ops.mx_quantize(torch.empty(0, 64, dtype=torch.bfloat16, device="cuda"), rowwise=True, layout=0)
    assert row.codes.numel() == 0


def test_retile_and_dequantise_roundtrip():
    ops = _ops()
    x = _activations(200, 320, seed=5)
    plain, _ = ops.mx_quantize(x.cuda(), rowwise=True, layout=0)
    tiled, _ = ops.mx_quantize(x.cuda(), rowwise=True, layout=1)
    assert torch.equal(ops.mx_retile(plain).scales, tiled.scales)
    d0, d1 = ops.mx_dequantize(plain), ops.mx_dequantize(tiled)
    assert torch.equal(d0, d1)
    want = OQ.round_to_bf16(OQ.dequantize_rowwise(plain.codes.cpu().numpy(), plain.scales.cpu().numpy()))
    assert np.array_equal(d0.float().cpu().numpy(), want)
    # quantise -> dequantise noise, the reference's own acceptance (tests/sanity_mxfp8_triton.py:49-52)
    rel = (d0.float().cpu() - x.float()).abs().max() / x.float().abs().max()
    assert rel < 0.10


def test_full_size_properties():
    """x [32768, 2048] (config 2): oracle on a 512-row slice, plus properties that hold at any size:
    the column form equals the row form of the transpose, dequantised values re-quantise to
    themselves, and |dequant - x| <= 2^(e-4) * ... bounded by one e4m3 half-step."""
    ops = _ops()
    x = _activations(32768, 2048, seed=42).cuda()
    row, col = ops.mx_quantize(x, rowwise=True, colwise=True, layout=0)
    sl = slice(13 * 512, 14 * 512)
    codes, scales = OQ.quantize_rowwise(x[sl].cpu().float().numpy())
    assert np.array_equal(row.codes[sl].cpu().numpy(), codes) and np.array_equal(row.scales[sl].cpu().numpy(), scales)
    rowT, _ = ops.mx_quantize(x.t().contiguous(), rowwise=True, layout=0)
    assert torch.equal(rowT.codes, col.codes) and torch.equal(rowT.scales, col.scales)
    deq = ops.mx_dequantize(row)
    again, _ = ops.mx_quantize(deq, rowwise=True, layout=0)   # representable values survive exactly
    assert torch.equal(ops.mx_dequantize(again), deq)
    # relative step of e4m3 is 2^-3; error <= half a step of the block's top binade
    step = torch.ldexp(torch.ones((), device="cuda"), row.scales.int() - 127 + 8 - 4)   # 2^(e+8) * 2^-4
    err = (deq.float() - x.float()).abs().view(32768, 64, 32).amax(dim=2)
    assert bool((err <= step).all())


@pytest.mark.parametrize("rows,cols", [(28288, 2048), (28416, 2048), (28448, 2048), (28416, 2016)])
def test_both_forms_equal_each_form_alone_around_the_resident_cta_rule(rows, cols):
    """3536, 3552, 3568 tiles of 128 x 128 (24 a SM is 3552), and a ragged last column tile."""
    ops = _ops()
    x = _activations(rows, cols, seed=rows).cuda()
    row, col = ops.mx_quantize(x, rowwise=True, colwise=True)
    for got, want in ((row, ops.mx_quantize(x, rowwise=True)[0]), (col, ops.mx_quantize(x, rowwise=False, colwise=True)[1])):
        assert torch.equal(got.codes, want.codes) and torch.equal(got.scales, want.scales)


def test_exponent_rule_against_the_references_expression_on_this_gpu(capsys):
    """The reference computes the block exponent as ceil(log2(amax) - log2(448)) in fp32 with the GPU's approximate
    log2 (mxfp8_gemm.py:118-120); the library uses the exact integer rule. Evaluate both on the device for EVERY
    positive finite bf16 value (a block maximum of bf16 data is one of them): any difference must be confined to
    block maxima whose mantissa is exactly 1.75 (the ceiling's edge), and is reported."""
    from anima_trainer_sm120_b200 import _lib
    bits = torch.arange(1, 0x7F80, dtype=torch.int32)                       # positive, finite, non-zero bf16 patterns
    amax = (bits << 16).view(torch.float32).cuda()
    n = amax.numel()
    by_rule = torch.empty(n, dtype=torch.int32, device="cuda")
    by_lg2 = torch.empty(n, dtype=torch.int32, device="cuda")
    _lib.check(_lib.load().anima_mx_exponent_probe(amax.data_ptr(), n, by_rule.data_ptr(), by_lg2.data_ptr(),
                                                   _lib.stream_ptr(torch.device("cuda"))))
    torch.cuda.synchronize()
    want = torch.from_numpy(OQ.exponent_exact(np.maximum(amax.cpu().numpy(), OQ.AMAX_FLOOR)))
    assert torch.equal(by_rule.cpu(), want)                                 # the kernel's rule is the oracle's
    diff = (by_rule != by_lg2).cpu()
    mant = bits & 0x7F
    edge = mant == 0x60                                                     # mantissa 1.75 exactly
    with capsys.disabled():
        print(f"\nexponent by rule vs ceil(lg2.approx(amax) - lg2.approx(448)) on this GPU: {int(diff.sum())} of {n} "
              f"bf16 block maxima differ; {int((diff & edge).sum())} of them have mantissa 1.75 "
              f"({int(edge.sum())} such values exist); binary exponents of those that differ: "
              f"{sorted(int(b >> 7) - 127 for b in bits[diff].tolist())}")
    assert not bool((diff & ~edge).any()), bits[diff & ~edge][:10].tolist()
