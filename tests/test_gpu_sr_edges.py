"""Stochastic rounding where it turns: random words at, one below and one above the threshold of each element, and the
extremes, for values at the ends of E2M1's ranges, against the oracle.  (Uniform words meet a threshold once in 2^32.)"""
import pytest
import torch

pytestmark = pytest.mark.gpu

from alto_b200 import _lib as L
from alto_b200 import _linear as E
from oracle import alto_oracle as O
from tests.helpers import to_u32_device

ENDS = [0.0, 0.25, 0.5, 0.75, 1.0, 1.25, 1.5, 1.75, 2.0, 2.5, 3.0, 3.5, 4.0, 5.0, 5.96875, 6.0, 6.25]


def _values(rows, cols, dtype, g):
    ends = torch.tensor(ENDS)
    pick = ends[torch.randint(0, len(ENDS), (rows, cols), generator=g)]
    steps = torch.randint(-1, 2, (rows, cols), generator=g)          # the end or a neighbour of the type
    bits = torch.int16 if dtype == torch.bfloat16 else torch.int32
    x = (pick.to(dtype).view(bits) + steps.to(bits)).clamp(min=0).to(bits).view(dtype).float()
    r = torch.rand(rows, cols, generator=g)
    x = torch.where(r < 0.3, torch.rand(rows, cols, generator=g) * torch.where(r < 0.15, 1.0, 6.0), x)
    x = torch.where((r >= 0.3) & (r < 0.35), torch.exp2(torch.randint(-36, 0, (rows, cols), generator=g).float()), x)
    x[:, ::16] = 6.0                                                 # block scales of 1 or 1.125
    return (x * torch.where(torch.rand(rows, cols, generator=g) < 0.5, -1.0, 1.0)).to(dtype)


def _words(v, g):
    """A word per quotient: the threshold of its rounding and its neighbours, all zeros, all ones."""
    a = v.abs()
    below = (a.double() * 2.0 ** 33).clamp(max=2.0 ** 34).long() % 2 ** 32       # a < 1: rounds up at and below it
    low = a.view(torch.int32).long() & 0x3FFFFF                                  # a >= 1: rounds up from 2^22 - low on
    at = torch.where(a < 1.0, below, 2 ** 22 - low + (torch.randint(0, 2 ** 10, a.shape, generator=g) << 22))
    kind = torch.randint(0, 5, a.shape, generator=g)
    out = torch.where(kind < 3, at + kind - 1, torch.where(kind == 3, 0, 2 ** 32 - 1))
    return out % 2 ** 32


@pytest.mark.parametrize("is_2d", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("fmt", [L.FMT_NVFP4, L.FMT_MXFP4])
@pytest.mark.parametrize("shape", [(64, 128), (96, 544)])
def test_words_at_the_thresholds(shape, fmt, dtype, is_2d):
    rows, cols = shape
    g = torch.Generator().manual_seed(0)
    x = _values(rows, cols, dtype, g)
    oracle, block = (O.quantize_nvfp4, 16) if fmt == L.FMT_NVFP4 else (O.quantize_mxfp4, 32)
    _, scales = oracle(x, block, -1, is_2d)
    q = scales.float() if fmt == L.FMT_NVFP4 else torch.exp2(scales.float() - 127.0)
    q = q.repeat_interleave(block, 1).repeat_interleave(block if is_2d else 1, 0)
    words = _words(x.float() / q, g)
    planes = torch.stack([words[:, 0::2], words[:, 1::2]])
    want = (O.quantize_nvfp4(x, 16, -1, is_2d, None, planes) if fmt == L.FMT_NVFP4
            else O.quantize_mxfp4(x, 32, -1, is_2d, planes))[0]
    sr = dict(rounding=L.ROUND_SR_BITS, rand_bits=to_u32_device(planes, "cuda"))
    if is_2d:
        got = [E.quant_2d(x.cuda(), fmt, None, True, False, sr)[0]]
    else:
        # along the rows; along the columns of the transposed matrix, with the words one by one and from a table
        got = [E.quant_rows(x.cuda(), fmt, None, sr), E.quant_cols(x.t().contiguous().cuda(), fmt, None, None, sr)]
        got.append(E.quant_cols(x.t().contiguous().cuda(), fmt, None, None, dict(sr, rand_tile=(rows, cols // 2))))
    for op in got:
        assert torch.equal(op.codes.cpu(), want.view(torch.uint8).reshape(rows, cols // 2))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("fmt", [L.FMT_NVFP4, L.FMT_MXFP4])
def test_words_of_the_slot_ordered_table_at_the_thresholds(fmt, dtype):
    """One tile of the table, so that each of its words belongs to one element."""
    g = torch.Generator().manual_seed(1)
    x = _values(64, 64, dtype, g)
    oracle, block = (O.quantize_nvfp4, 16) if fmt == L.FMT_NVFP4 else (O.quantize_mxfp4, 32)
    _, scales = oracle(x, block, -1)
    q = scales.float() if fmt == L.FMT_NVFP4 else torch.exp2(scales.float() - 127.0)
    words = _words(x.float() / q.repeat_interleave(block, 1), g)
    planes = torch.stack([words[:, 0::2], words[:, 1::2]])
    want = (O.quantize_nvfp4(x, 16, -1, False, None, planes) if fmt == L.FMT_NVFP4
            else O.quantize_mxfp4(x, 32, -1, False, planes))[0]
    # [position][row]; without a transform slots are positions
    got = E.quant_cols(x.t().contiguous().cuda(), fmt, None, None,
                       dict(rounding=L.ROUND_SR_SLOTS, rand_bits=to_u32_device(words.t().contiguous(), "cuda"),
                            rand_tile=L.SLOTS_TILE))
    assert torch.equal(got.codes.cpu(), want.view(torch.uint8).reshape(64, 32))
