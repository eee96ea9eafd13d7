"""The two-level GEMM where its rings wrap and its CTAs take several tiles, against float64: factors that differ from
chunk to chunk, odd chunk counts and a short last chunk, an absent second half, both tile widths, K ranges of uneven
length, groups without an expert."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from alto_b200 import _lib as L
from alto_b200 import _linear as E

E2M1 = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], dtype=torch.float64)


class Random:
    """An operand [rows, k] of random codes, block exponents and factor codes, and the values it stands for."""

    def __init__(self, rows, k, seed, tiles=False):
        g = torch.Generator(device="cuda").manual_seed(seed)
        nc = -(-k // 128)
        draw = lambda low, high, *shape: torch.randint(low, high, shape, generator=g, device="cuda", dtype=torch.uint8)
        self.codes, exps = draw(0, 256, rows, k // 2), draw(122, 132, rows, k // 32)
        self.scales = E.pack_plain_scales(exps, rows, False, 32)
        f = draw(0, 256, -(-rows // 128) if tiles else rows, nc)
        self.macro = L.MacroScale(f, nc, 1, 7 if tiles else 0)
        nibbles = torch.stack([self.codes & 15, self.codes >> 4], -1).reshape(rows, k).long()
        v = torch.where(nibbles >= 8, -1.0, 1.0) * E2M1.cuda()[nibbles & 7]
        v *= torch.exp2(exps.double() - 127.0).repeat_interleave(32, 1)
        per_row = f.repeat_interleave(128, 0)[:rows] if tiles else f
        self.values = v / (1.0 + per_row.double() / 256.0).repeat_interleave(128, 1)[:, :k]


def _near(got, a, b):
    # fp32 sums of a chunk (the tensor core may truncate: two bits), of the chunks, two roundings of the factors
    chunks = -(-a.shape[1] // 128)
    bound = (chunks + 16) * 2.0 ** -22 * (a.abs() @ b.abs().t())
    assert ((got.double() - a @ b.t()).abs() <= bound).all()


# (k = 2880: 23 chunks, the last of 64.)  Narrow tiles: few; several per CTA, the last one half.  Wide tiles: several
# per CTA, the last column tile without a second half.
SHAPES = [(96, 160), (2304, 2336), (3712, 2400)]


@pytest.mark.parametrize("tiles", [False, True])
@pytest.mark.parametrize("k", [32, 640, 2880])
@pytest.mark.parametrize("shape", SHAPES)
def test_dense(shape, k, tiles):
    m, n = shape
    a, b = Random(m, k, 1), Random(n, k, 2, tiles)
    out = torch.empty(m, n, dtype=torch.float32, device="cuda")
    L.gemm_mxfp4_two_level(m, n, k, a.codes, a.scales, a.macro, b.codes, b.scales, b.macro, out)
    _near(out, a.values, b.values)
    # a column range of its own has fewer tiles, hence other tile widths, and the same bits
    part = torch.empty(m, 128, dtype=torch.float32, device="cuda")
    L.gemm_mxfp4_two_level(m, 128, k, a.codes, a.scales, a.macro, b.codes, b.scales, b.macro, part)
    assert torch.equal(part, out[:, :128])
    half = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    L.gemm_mxfp4_two_level(m, n, k, a.codes, a.scales, a.macro, b.codes, b.scales, b.macro, half, 0.5)
    assert torch.equal(half, (out * 0.5).bfloat16())


@pytest.mark.parametrize("shape,counts", [((96, 160), [128]), ((1152, 1312), [384, 0, 640, 128, 0, 1152, 256]),
                                          ((3712, 2400), [1408, 0, 1152])])
def test_k_ranges(shape, counts):
    m, n = shape
    total, ends = sum(counts), torch.tensor(counts).cumsum(0).to(torch.int32).cuda()
    a, b = Random(m, total, 3), Random(n, total, 4)
    out = torch.full((len(counts), m, n), 7.0, dtype=torch.float32, device="cuda")
    L.gemm_mxfp4_two_level(m, n, total, a.codes, a.scales, a.macro, b.codes, b.scales, b.macro, out, k_offs=ends,
                           num_experts=len(counts))
    start = 0
    for e, end in enumerate(ends.tolist()):
        _near(out[e], a.values[:, start:end], b.values[:, start:end])
        start = end


@pytest.mark.parametrize("tiles", [False, True])
@pytest.mark.parametrize("k", [640, 2880])
@pytest.mark.parametrize("groups,n", [([1, 0], 160), ([2, 0, 0, -1, 1, 2, -1], 416), ([0, 1] * 12, 2336)])
def test_row_groups(groups, n, k, tiles):
    m, n_exp = 128 * len(groups), 3
    a = Random(m, k, 5)
    bs = [Random(n, k, 6 + e, tiles) for e in range(n_exp)]
    macro = torch.stack([b.macro.codes for b in bs])
    f = L.MacroScale(macro, bs[0].macro.row_stride, 1, bs[0].macro.row_shift, macro[0].numel())
    out = torch.full((m, n), 7.0, dtype=torch.float32, device="cuda")
    L.gemm_mxfp4_two_level(m, n, k, a.codes, a.scales, a.macro, torch.cat([b.codes for b in bs]),
                           torch.cat([b.scales for b in bs]), f, out,
                           group_expert=torch.tensor(groups, dtype=torch.int32, device="cuda"), num_experts=n_exp)
    for i, e in enumerate(groups):
        rows = slice(128 * i, 128 * i + 128)
        if e < 0:
            assert (out[rows] == 0).all()
        else:
            _near(out[rows], a.values[rows], bs[e].values)


@pytest.mark.parametrize("n", [2304 + 32, 2304 + 160])
@pytest.mark.parametrize("k", [640, 2880])
def test_wide_tiles_of_row_groups(n, k):
    # 18 row tiles: tiles of 192 columns, whose scales of B begin on a block of 128 rows or in its middle; the last
    # tile ends before its second block, or in it, and reads on into the next expert's rows
    groups, n_exp = [0, 1] * 9, 2
    a = Random(128 * len(groups), k, 15)
    bs = [Random(n, k, 16 + e, True) for e in range(n_exp)]
    macro = torch.stack([b.macro.codes for b in bs])
    f = L.MacroScale(macro, bs[0].macro.row_stride, 1, 7, macro[0].numel())
    out = torch.empty(128 * len(groups), n, dtype=torch.float32, device="cuda")
    L.gemm_mxfp4_two_level(out.shape[0], n, k, a.codes, a.scales, a.macro, torch.cat([b.codes for b in bs]),
                           torch.cat([b.scales for b in bs]), f, out,
                           group_expert=torch.tensor(groups, dtype=torch.int32, device="cuda"), num_experts=n_exp)
    for i, e in enumerate(groups):
        rows = slice(128 * i, 128 * i + 128)
        _near(out[rows], a.values[rows], bs[e].values)


@pytest.mark.parametrize("shape,counts", [((2304, 2336), [128] * 16), ((2304, 2336), [128, 128, 256, 128, 384, 128, 128, 0] * 3),
                                          ((5760, 2880), [128] * 16)])
def test_single_chunk_stages(shape, counts):
    # dozens of tiles a CTA, most of them one chunk in a stage of its own: the ring of factors is reused at its closest
    m, n = shape
    total, ends = sum(counts), torch.tensor(counts).cumsum(0).to(torch.int32).cuda()
    a, b = Random(m, total, 31), Random(n, total, 32)
    out = torch.full((len(counts), m, n), 7.0, dtype=torch.float32, device="cuda")
    L.gemm_mxfp4_two_level(m, n, total, a.codes, a.scales, a.macro, b.codes, b.scales, b.macro, out, k_offs=ends,
                           num_experts=len(counts))
    start = 0
    for e, end in enumerate(ends.tolist()):
        _near(out[e], a.values[:, start:end], b.values[:, start:end])
        start = end


@pytest.mark.parametrize("k", [32, 128])
def test_single_chunk_stages_dense(k):
    m, n = 9216, 2592                              # ten tiles a CTA
    a, b = Random(m, k, 33), Random(n, k, 34)
    out = torch.empty(m, n, dtype=torch.float32, device="cuda")
    L.gemm_mxfp4_two_level(m, n, k, a.codes, a.scales, a.macro, b.codes, b.scales, b.macro, out)
    _near(out, a.values, b.values)
