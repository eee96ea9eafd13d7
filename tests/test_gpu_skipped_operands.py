"""Operands that only a gradient needs are not made where no gradient can be asked for."""
import contextlib

import pytest
import torch

pytestmark = pytest.mark.gpu

from alto_b200 import _lib as L
from alto_b200 import mxfp4, mxfp8, nvfp4

CALLS = {"nvfp4": lambda x, w, w2d: nvfp4._to_nvfp4_then_scaled_mm(x, w, False, w2d, True, use_outer_scale=True,
                                                                   use_hadamard=True),
         "mxfp4": lambda x, w, w2d: mxfp4._to_mxfp4_then_scaled_mm(x, w, False, w2d, True, False, "none", True),
         "mxfp8": lambda x, w, w2d: mxfp8._to_mxfp8_then_scaled_mm(x, w, "e4m3", False, False, w2d)}


def _launches(monkeypatch, call):
    seen = []
    with monkeypatch.context() as patch:
        for name in ("amax", "quantize_rowwise", "quantize_colwise", "quantize_2d", "gemm_blockscaled"):
            real = getattr(L, name)

            def wrapped(*args, _name=name, _real=real, **kw):
                transposed = _name == "quantize_2d" and args[3] is not None
                rotated = kw.get("rht") is not None or (_name == "amax" and len(args) > 4 and args[4] is not None)
                seen.append((_name, transposed, rotated))
                return _real(*args, **kw)

            patch.setattr(L, name, wrapped)
        y = call()
    return seen, y.detach().clone()


@pytest.mark.parametrize("mode", [torch.no_grad, torch.inference_mode])
@pytest.mark.parametrize("weight_2d", [False, True])
@pytest.mark.parametrize("recipe", list(CALLS))
def test_evaluation_of_parameters(monkeypatch, recipe, weight_2d, mode):
    """Parameters keep requires_grad in an evaluation pass: it launches what tensors without it launch."""
    g = torch.Generator().manual_seed(0)
    x = torch.randn(128, 192, generator=g).bfloat16().cuda()
    w = (torch.randn(160, 192, generator=g) * 0.02).bfloat16().cuda()

    def run(context, x, w):
        with context():
            return _launches(monkeypatch, lambda: CALLS[recipe](x, w, weight_2d))

    plain, y0 = run(contextlib.nullcontext, x, w)
    evaluated, y1 = run(mode, x.clone().requires_grad_(True), torch.nn.Parameter(w.clone()))
    assert evaluated == plain
    assert torch.equal(y0, y1)
    trained, y2 = run(contextlib.nullcontext, x.clone().requires_grad_(True), torch.nn.Parameter(w.clone()))
    assert trained != plain and torch.equal(y0, y2)


def test_evaluation_of_a_converted_module(monkeypatch):
    from alto_b200 import dispatch
    config = dispatch.TrainingOpConfig(precision="mxfp8_e4m3", use_2dblock_x=False, use_2dblock_w=True, use_hadamard=False,
                                       use_sr_grad=False, use_dge=False)
    layer = torch.nn.Linear(192, 160, bias=False, dtype=torch.bfloat16, device="cuda")
    w = layer.weight.detach().clone()
    x = torch.randn(128, 192, generator=torch.Generator().manual_seed(0)).bfloat16().cuda()
    plain, y0 = _launches(monkeypatch, lambda: CALLS["mxfp8"](x, w, True))
    dispatch.swap_params(layer, config=config)
    with torch.no_grad():
        evaluated, y1 = _launches(monkeypatch, lambda: layer(x))
    assert layer.weight.requires_grad and evaluated == plain and torch.equal(y0, y1)
    trained, _ = _launches(monkeypatch, lambda: layer(x))
    assert trained != plain


@pytest.mark.parametrize("weight_2d", [False, True])
@pytest.mark.parametrize("recipe", list(CALLS))
def test_forward_of_a_frozen_side(monkeypatch, recipe, weight_2d):
    """Only dX asked for: X is not quantised along the tokens.  Only dW: the weight has no second packing."""
    x, w = torch.randn(128, 192).bfloat16().cuda(), torch.randn(160, 192).bfloat16().cuda()

    def seen(need_x, need_w):
        launches, _ = _launches(monkeypatch, lambda: CALLS[recipe](x.clone().requires_grad_(need_x),
                                                                   w.clone().requires_grad_(need_w), weight_2d))
        return (sum(name == "quantize_colwise" for name, _, _ in launches), sum(t for _, t, _ in launches))

    transposed = int(weight_2d)                       # 2-D blocks: the second packing; 1-D: a column-wise launch
    assert seen(True, True) == (2 - transposed, transposed)
    assert seen(True, False) == (1 - transposed, transposed)
    assert seen(False, True) == (1, 0)
    assert seen(False, False) == (0, 0)
