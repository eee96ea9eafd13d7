"""Row-wise quantizer with a periodic table of random words (rows a period apart share them) against the same words
written out for every element."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from alto_b200 import _lib as L


def _quantise(x, fmt, outer, macro, **words):
    rows, cols = x.shape
    codes = torch.empty(rows, cols // 2, dtype=torch.uint8, device="cuda")
    packed = torch.full((-(-rows // 128) * 128, -(-cols // L.block_of(fmt) // 4) * 4), 0, dtype=torch.uint8, device="cuda")
    factors = torch.empty(rows, -(-cols // 128), dtype=torch.uint8, device="cuda") if macro else None
    L.quantize_rowwise(x, fmt, codes, None, packed, outer_scale=outer, rounding=L.ROUND_SR_BITS, macro_codes=factors, **words)
    return [codes, packed] + ([factors] if macro else [])


@pytest.mark.parametrize("rows,cols", [(1, 64), (31, 64), (64, 32), (65, 512), (130, 544), (255, 96), (256, 1024), (321, 1056), (4099, 64)])
@pytest.mark.parametrize("fmt,dtype,macro", [(L.FMT_MXFP4, torch.bfloat16, False), (L.FMT_MXFP4, torch.bfloat16, True),
                                             (L.FMT_MXFP4, torch.float32, False), (L.FMT_NVFP4, torch.bfloat16, False),
                                             (L.FMT_NVFP4, torch.float32, False)])
@pytest.mark.parametrize("special", [False, True])
def test_equals_words_for_every_element(rows, cols, fmt, dtype, macro, special):
    g = torch.Generator(device="cuda").manual_seed(rows * 7 + cols)
    x = torch.randn(rows, cols, generator=g, device="cuda") * torch.logspace(-6, 6, cols, device="cuda")
    x[:, 5], x[:, 6], x[rows // 2] = 0.0, -0.0, 0.0
    if special:
        x[rows - 1, 0], x[rows // 3, 1], x[0, 2] = float("nan"), float("inf"), 1.0e-39
    x = x.to(dtype)
    tile = L.sr_tile_dims(rows, cols)
    table = torch.randint(-2 ** 31, 2 ** 31, (2, *tile), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    table[0, 0, :4] = torch.tensor([0, -1, 1, 0x3FFFFF], dtype=torch.int32, device="cuda")
    r, c = torch.arange(rows, device="cuda") % tile[0], torch.arange(cols // 2, device="cuda") % tile[1]
    planes = table[:, r][:, :, c].contiguous()
    outer = torch.tensor([0.37], device="cuda") if fmt == L.FMT_NVFP4 else None
    one = _quantise(x, fmt, outer, macro, rand_bits=table, rand_tile=tile)
    two = _quantise(x, fmt, outer, macro, rand_bits=planes)
    assert all(torch.equal(a, b) for a, b in zip(one, two))


@pytest.mark.parametrize("rows,cols,tile", [(96, 65536, None), (31, 131072, None), (321, 65536 + 32, None), (40, 544, (200_000, 8)),
                                            (5, 4128, (3, 16))])
@pytest.mark.parametrize("fmt,dtype,macro", [(L.FMT_MXFP4, torch.bfloat16, False), (L.FMT_MXFP4, torch.bfloat16, True),
                                             (L.FMT_MXFP4, torch.float32, False), (L.FMT_NVFP4, torch.bfloat16, False),
                                             (L.FMT_NVFP4, torch.float32, False)])
@pytest.mark.parametrize("special", [False, True])
def test_few_rows_equal_words_for_every_element(rows, cols, tile, fmt, dtype, macro, special):
    # wide enough that the rows of a task are neighbours, each with words of its own; a table far longer than the rows
    tile = tile or L.sr_tile_dims(rows, cols)
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = torch.randn(rows, cols, generator=g, device="cuda") * torch.logspace(-6, 6, cols, device="cuda")
    if special:
        x[rows - 1, 0], x[rows // 3, 1], x[0, 2] = float("nan"), float("inf"), -0.0
    x = x.to(dtype)
    table = torch.randint(-2 ** 31, 2 ** 31, (2, *tile), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    r, c = torch.arange(rows, device="cuda") % tile[0], torch.arange(cols // 2, device="cuda") % tile[1]
    planes = table[:, r][:, :, c].contiguous()
    outer = torch.tensor([0.37], device="cuda") if fmt == L.FMT_NVFP4 else None
    one = _quantise(x, fmt, outer, macro, rand_bits=table, rand_tile=tile)
    two = _quantise(x, fmt, outer, macro, rand_bits=planes)
    assert all(torch.equal(a, b) for a, b in zip(one, two))
