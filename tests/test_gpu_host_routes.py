"""Routes that spare host work against the general ones: the backward behind one call, matrices dequantised as they are;
the maximum of tensors at the sizes where its loads a thread change."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from alto_b200 import _lib as L
from alto_b200 import _linear as E
from alto_b200 import _quant as Q
from alto_b200 import mxfp4, mxfp8, nvfp4

CALLS = {
    "nvfp4": lambda x, w, w2d, sr, rht: nvfp4._to_nvfp4_then_scaled_mm(x, w, False, w2d, sr, use_outer_scale=True, use_hadamard=rht),
    "nvfp4_plain": lambda x, w, w2d, sr, rht: nvfp4._to_nvfp4_then_scaled_mm(x, w, False, w2d, sr, use_hadamard=rht),
    "mxfp4": lambda x, w, w2d, sr, rht: mxfp4._to_mxfp4_then_scaled_mm(x, w, False, w2d, sr, False, "none", rht),
    "mxfp8": lambda x, w, w2d, sr, rht: mxfp8._to_mxfp8_then_scaled_mm(x, w, "e4m3", False, False, w2d),
}


@pytest.mark.parametrize("recipe,w2d,sr,rht", [("nvfp4", True, True, 16), ("nvfp4", False, False, 0), ("nvfp4_plain", True, True, 0),
                                               ("mxfp4", True, True, 16), ("mxfp4", False, True, 0), ("mxfp8", True, False, 0)])
@pytest.mark.parametrize("m,k,n,dtype", [(32, 32, 32, torch.bfloat16), (96, 160, 224, torch.float32), (320, 288, 96, torch.bfloat16)])
def test_backward_behind_one_call(monkeypatch, recipe, w2d, sr, rht, m, k, n, dtype):
    # (views of fewer than 64 rows or columns have a smaller table of random words, whole ones the slot-ordered one)
    def grads(one_call, ask, strided):
        if rht:
            nvfp4.HadamardFactory.configure(block_size=rht, randomized=True, dtype=torch.float32, seed=5)
        torch.default_generator.manual_seed(7)
        g = torch.Generator(device="cuda").manual_seed(3)
        x = torch.randn(2, m // 2, k, generator=g, device="cuda").to(dtype).requires_grad_("x" in ask)
        w = (torch.randn(n, k, generator=g, device="cuda") * 0.02).to(dtype).requires_grad_("w" in ask)
        dy = (torch.randn(2, m // 2, 2 * n, generator=g, device="cuda") * 1e-3).to(dtype)
        dy = dy[..., :n] if strided else dy[..., :n].contiguous()
        routes = []
        real = L.linear_backward
        with monkeypatch.context() as patch:
            patch.setattr(L, "linear_backward", lambda *a: routes.append(1) or real(*a))
            if not one_call:
                patch.setattr(E, "one_call_backward", lambda *a: False)
            y = CALLS[recipe](x, w, w2d, sr, bool(rht))
            out = torch.autograd.grad(y, [t for t in (x, w) if t.requires_grad], dy)
        assert len(routes) == int(one_call)
        return (y.detach(), *out, torch.default_generator.get_state().cuda())

    for ask, strided in (("xw", False), ("xw", True), ("x", False), ("w", False)):
        for a, b in zip(grads(True, ask, strided), grads(False, ask, strided)):
            assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b)


@pytest.mark.parametrize("fmt", [L.FMT_NVFP4, L.FMT_MXFP4, L.FMT_MXFP8_E4M3, L.FMT_MXFP8_E5M2])
@pytest.mark.parametrize("is_2d", [False, True])
def test_a_matrix_is_dequantised_as_it_is(fmt, is_2d):
    rows, cols, block = (96 if is_2d else 37), 160, L.block_of(fmt)
    x = torch.randn(rows, cols, generator=torch.Generator().manual_seed(1)).cuda()
    outer = torch.full((1,), 0.01, device="cuda") if fmt == L.FMT_NVFP4 else None
    codes, scales = Q.quantize(x, fmt, -1, is_2d, outer_scale=outer)
    batched = Q.quantize(x[None], fmt, -1, is_2d, outer_scale=outer)
    assert all(a.dtype == b.dtype and torch.equal(a.view(torch.uint8), b[0].view(torch.uint8)) for a, b in zip((codes, scales), batched))
    half = scales.bfloat16() if fmt == L.FMT_NVFP4 else scales       # E4M3 values, exact in bf16
    for c, s in ((codes, scales), (codes.t().contiguous().t(), scales.t().contiguous().t()), (codes, half)):
        for dtype in (torch.float32, torch.bfloat16):
            got = Q.dequantize(c, s, fmt, -1, is_2d, dtype, outer)
            want = Q.dequantize(codes[None], scales[None], fmt, -1, is_2d, dtype, outer)[0]
            assert got.dtype == dtype and got.shape == (rows, cols) and torch.equal(got, want)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,cols,pitch", [(1, 8, 8), (37, 2056, 2056), (1200, 8200, 8200), (1187, 8192, 8208), (2411, 8200, 8208),
                                             (5000, 8200, 8200)])
def test_maximum_wherever_it_lies(rows, cols, pitch, dtype):
    # one load a thread, a few, four (1184 blocks of 256 threads and more), eight
    x = torch.zeros(rows, pitch, dtype=dtype, device="cuda")[:, :cols]
    bits, outer, scratch = torch.empty(2, dtype=torch.int32, device="cuda"), torch.empty(2, device="cuda"), E.amax_scratch(x.device)
    for i, (r, c) in enumerate([(0, 0), (rows - 1, cols - 1), (rows // 2, cols // 3), (rows - 1, 0), (0, cols - 1)]):
        x[r, c] = -(i + 1.5)
        L.amax(x, bits, outer, scratch)
        assert bits.view(torch.float32)[0].item() == i + 1.5


@pytest.mark.parametrize("fmt", [L.FMT_NVFP4, L.FMT_MXFP4, L.FMT_MXFP8_E4M3])
@pytest.mark.parametrize("is_2d,pad", [(False, 91), (True, 6)])
def test_scales_with_rows_behind_the_codes(fmt, is_2d, pad):
    # buffers of scales are padded by some callers; too few are refused
    rows, cols, block = (96 if is_2d else 37), 160, L.block_of(fmt)
    x = torch.randn(rows, cols, generator=torch.Generator().manual_seed(2)).cuda()
    codes, scales = Q.quantize(x, fmt, -1, is_2d)
    want = Q.dequantize(codes, scales, fmt, -1, is_2d, torch.float32)
    more = torch.cat([scales, torch.ones(pad, scales.shape[1], device="cuda").to(scales.dtype)])
    if is_2d:
        more = more[:2 * scales.shape[0]]
    assert torch.equal(Q.dequantize(codes, more, fmt, -1, is_2d, torch.float32), want)
    with pytest.raises(RuntimeError):
        Q.dequantize(codes, scales[:-1], fmt, -1, is_2d, torch.float32)


@pytest.mark.parametrize("dtype,cols", [(torch.bfloat16, 2048), (torch.float32, 1024)])      # 256 loads a row
@pytest.mark.parametrize("steps,more", [(1, 1), (4, 0), (4, 1), (9, -1), (9, 0)])
def test_maximum_where_the_loads_of_a_thread_change(dtype, cols, steps, more):
    blocks = torch.cuda.get_device_properties(0).multi_processor_count * 8
    rows = blocks * steps + more
    x = torch.zeros(rows, cols, dtype=dtype, device="cuda")
    bits, outer, scratch = torch.empty(2, dtype=torch.int32, device="cuda"), torch.empty(2, device="cuda"), E.amax_scratch(x.device)
    for i, (r, c) in enumerate([(0, 0), (rows - 1, cols - 1), (rows - 1, 0), (blocks * 8 % rows, cols // 2), (blocks * 4 % rows, 3)]):
        x[r, c] = -(i + 1.5)
        L.amax(x, bits, outer, scratch)
        assert bits.view(torch.float32)[0].item() == i + 1.5
