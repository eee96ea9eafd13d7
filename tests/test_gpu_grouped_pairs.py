"""Rows grouped by expert on CTA pairs: every group of 128 rows against the same rows multiplied alone (another kernel)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from alto_b200 import _lib as L
from alto_b200 import _linear as E

# pairs of one expert, of two, with a group of none before, behind or both, a lone last group; units over several warps
GROUPS = [[0, 0, 0, 1], [1, 0, 0, 1, -1, 1, 0, -1, -1, -1, 0], [0] * 7 + [2] * 9 + [1] + [-1] * 3, [i // 5 % 3 for i in range(141)] + [-1]]


@pytest.mark.parametrize("fmt", [L.FMT_NVFP4, L.FMT_MXFP4, L.FMT_MXFP8_E4M3])
@pytest.mark.parametrize("n,k", [(160, 96), (544, 1056)])
@pytest.mark.parametrize("groups", GROUPS)
def test_groups_equal_their_rows_alone(groups, n, k, fmt):
    m, n_exp = 128 * len(groups), max(groups) + 1
    if m < 512 * n_exp:
        groups = groups * 3
        m = 128 * len(groups)
    assert m >= 512 * n_exp                      # as many rows as the rule asks for
    g = torch.Generator(device="cuda").manual_seed(k + len(groups))
    x = torch.randn(m, k, generator=g, device="cuda").bfloat16()
    w = torch.randn(n_exp * n, k, generator=g, device="cuda").bfloat16()
    outer = torch.tensor([0.5], device="cuda") if fmt == L.FMT_NVFP4 else None
    a = E.quant_rows(x, fmt, outer, E.RTN)
    bs = [E.quant_rows(w[e * n:(e + 1) * n], fmt, outer, E.RTN) for e in range(n_exp)]
    codes, scales = torch.cat([b.codes for b in bs]), torch.cat([b.scales for b in bs])
    ids = torch.tensor(groups, dtype=torch.int32, device="cuda")
    block = a.scales.numel() // len(groups)
    for dtype in (torch.bfloat16, torch.float32):
        out = torch.full((m, n), 7.0, dtype=dtype, device="cuda")
        L.grouped_gemm_blockscaled(fmt, fmt, m, n, k, n_exp, a.codes, a.scales, codes, scales, ids, out, outer, outer)
        for i, e in enumerate(groups):
            rows = slice(128 * i, 128 * i + 128)
            if e < 0:
                assert (out[rows] == 0).all()
                continue
            want = torch.empty(128, n, dtype=dtype, device="cuda")
            L.gemm_blockscaled(fmt, fmt, 128, n, k, a.codes[rows], a.scales[block * i:block * (i + 1)], bs[e].codes,
                               bs[e].scales, want, outer, outer)
            assert torch.equal(out[rows], want)


# the same over as many tiles as make pairs the faster ones, whatever the runs; 17 experts of an odd number of groups
@pytest.mark.parametrize("fmt", [L.FMT_NVFP4, L.FMT_MXFP4, L.FMT_MXFP8_E4M3])
@pytest.mark.parametrize("k", [96, 1056])
@pytest.mark.parametrize("groups", [g * (-(-160 // len(g))) for g in GROUPS] + [[i // 9 for i in range(153)]])
def test_many_groups_equal_their_rows_alone(groups, k, fmt):
    test_groups_equal_their_rows_alone(groups, 1056, k, fmt)
