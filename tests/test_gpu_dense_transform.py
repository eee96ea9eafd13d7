"""The 32-point transform inside the column-wise quantizer against the transform's own kernel in front of it."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from alto_b200 import _lib as L
from alto_b200 import _linear as E
from alto_b200 import _two_level as T
from alto_b200.hadamard import HadamardFactory, HadamardTransform

MX = L.FMT_MXFP4


def _transform(seed):
    HadamardFactory.configure(block_size=32, randomized=True, dtype=torch.float32, seed=seed)
    return HadamardFactory.create_transform("cuda")


def _same(a, b):
    pairs = [(a.codes, b.codes), (a.scales, b.scales)] + ([(a.macro.codes, b.macro.codes)] if a.macro is not None else [])
    assert all(torch.equal(x, y) for x, y in pairs)


@pytest.mark.parametrize("rows,cols,pitch", [(32, 32, 32), (96, 40, 48), (128, 64, 64), (160, 200, 200), (4128, 72, 96), (256, 320, 320)])
@pytest.mark.parametrize("clip,uos", [("none", False), ("static", True), ("dynamic", False)])
@pytest.mark.parametrize("sr", [False, True])
def test_equals_transform_then_quantize(monkeypatch, rows, cols, pitch, clip, uos, sr):
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = (torch.randn(rows, pitch, generator=g, device="cuda") * 3).bfloat16()[:, :cols]
    x[:32, 3] = 0
    x[rows - 1, 0], x[rows // 2, 1], x[5, 2] = float("nan"), float("inf"), -3.0e38
    transform, calls = _transform(7), []
    real = HadamardTransform.__call__
    monkeypatch.setattr(HadamardTransform, "__call__", lambda self, *a, **k: calls.append(1) or real(self, *a, **k))
    for quantise in (lambda s: E.cols_operand(x, MX, False, None, None, transform, s, uos, clip),
                     lambda s: T.cols_operand(x, uos, clip, s, transform)):
        words = E.RTN
        if sr:
            torch.default_generator.manual_seed(3)
            words = E.sr_args_cols(True, "dy_m", cols, rows, x.device)
        in_quantizer = words["rounding"] in (L.ROUND_RTN, L.ROUND_SR_SLOTS)   # whole tables of words, or none
        calls.clear()
        one = quantise(words)
        assert len(calls) == int(not in_quantizer)
        with monkeypatch.context() as patch:
            patch.setattr(E, "dense_in_quantizer", lambda *a: None)
            two = quantise(words)
        _same(one, two)


def test_transposed_rows_are_copied_as_before():
    x = torch.randn(64, 96, device="cuda").bfloat16()
    transform = _transform(5)
    _same(E.cols_operand(x.t(), MX, False, None, None, transform, E.RTN),
          E.cols_operand(x.t().contiguous(), MX, False, None, None, transform, E.RTN))


def test_other_formats_and_types_take_the_separate_kernel():
    transform = _transform(1)
    bf16, fp32 = torch.zeros(64, 64, dtype=torch.bfloat16, device="cuda"), torch.zeros(64, 64, device="cuda")
    assert E.dense_in_quantizer(bf16, transform, MX, E.RTN) is not None
    for t, fmt, sr in ((fp32, MX, E.RTN), (bf16, L.FMT_NVFP4, E.RTN), (bf16[:40], MX, E.RTN), (bf16.t(), MX, E.RTN),
                       (bf16[:, 2:34], MX, E.RTN), (bf16[:1].expand(64, 64), MX, E.RTN),
                       (torch.empty_strided((64, 64), (68, 1), dtype=torch.bfloat16, device="cuda"), MX, E.RTN),
                       (bf16, MX, dict(rounding=L.ROUND_SR_BITS))):
        assert E.dense_in_quantizer(t, transform, fmt, sr) is None
    codes = torch.empty(64, 32, dtype=torch.uint8, device="cuda")
    with pytest.raises(L.Altob200Error):
        L.quantize_colwise(fp32, MX, codes, torch.empty(64, 2, dtype=torch.uint8, device="cuda"), dense=transform.device_matrix(fp32.device))
