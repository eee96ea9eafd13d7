"""The dequantizer against the same values spelled out with tensor operations, at sizes around its vectors, blocks and
grid: fewer vectors than threads, one vector per thread, several, and a remainder."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from alto_b200 import _lib as L
from alto_b200 import _quant as Q

E2M1 = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0])


@pytest.mark.parametrize("is_2d", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("fmt", [L.FMT_NVFP4, L.FMT_MXFP4, L.FMT_MXFP8_E4M3, L.FMT_MXFP8_E5M2])
# 303104 threads at 148 SMs: the last two shapes give some of them one vector more than others
@pytest.mark.parametrize("shape", [(32, 32), (96, 160), (1184, 2048), (2400, 4128)])
def test_dequantized_values(shape, fmt, dtype, is_2d):
    rows, cols = shape
    block = L.block_of(fmt)
    g = torch.Generator().manual_seed(1)
    scale_shape = (rows // block if is_2d else rows, cols // block)
    if fmt == L.FMT_NVFP4:
        scales = torch.randint(1, 448, scale_shape, generator=g).float()
        factor = scales
    else:
        scales = torch.randint(100, 150, scale_shape, generator=g, dtype=torch.uint8)
        factor = torch.exp2(scales.float() - 127.0)
    if L.is_fp4(fmt):
        codes = torch.randint(0, 256, (rows, cols // 2), generator=g, dtype=torch.uint8)
        nibbles = torch.stack([codes & 15, codes >> 4], -1).reshape(rows, cols).long()
        values = torch.where(nibbles >= 8, -1.0, 1.0) * E2M1[nibbles & 7]
    else:
        f8 = torch.float8_e5m2 if fmt == L.FMT_MXFP8_E5M2 else torch.float8_e4m3fn
        codes = (torch.randn(rows, cols, generator=g) * 50).to(f8).view(torch.uint8)
        values = codes.view(f8).float()
    if is_2d:
        factor = factor.repeat_interleave(block, 0)
    want = (values * factor.repeat_interleave(block, 1)).to(dtype)
    got = Q.dequantize(codes.cuda(), scales.cuda(), fmt, -1, is_2d, dtype, None)
    assert torch.equal(got.cpu(), want)
