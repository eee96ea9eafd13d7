"""Calls at the edge of what the host functions and the C interface take."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from alto_b200 import _lib as L
from alto_b200 import _linear as E
from alto_b200 import _two_level as T


def test_amax_scratch_of_the_current_device():
    buf = E.amax_scratch(torch.device("cuda"))
    assert buf.is_cuda and buf.numel() * 4 >= L.AMAX_SCRATCH_BYTES and (buf == 0).all()
    assert E.amax_scratch(torch.device("cuda", torch.cuda.current_device())) is buf


def test_run_ends_are_a_vector():
    from alto_b200.grouped import group_experts_from_offsets
    offs = torch.tensor([[128, 256]], dtype=torch.int32)
    for t in (offs, offs.cuda()):
        with pytest.raises(RuntimeError):
            group_experts_from_offsets(t, 256)


class _Strided(L.MacroScale):
    """Factor codes whose row r starts ``first + r * row_stride`` bytes into a buffer."""

    __slots__ = ("first",)

    def desc(self):
        d = super().desc()
        d.codes += self.first
        return d


@pytest.mark.parametrize("m,n,stride", [(130, 96, "reversed"), (256, 416, "reversed"), (130, 96, "beyond 32 bits")])
def test_two_level_factors_with_any_row_stride(m, n, stride):
    k = 384
    g = torch.Generator().manual_seed(0)
    a = T.rows_operand(torch.randn(m, k, generator=g).bfloat16().cuda(), False)
    b = T.rows_operand(torch.randn(n, k, generator=g).bfloat16().cuda(), False)

    def moved(op):
        rows, nc = op.macro.codes.shape
        if stride == "reversed":
            scale = _Strided(op.macro.codes.flip(0).contiguous(), -nc, 1, 0)
            scale.first = (rows - 1) * nc
        else:
            pitch = (1 << 32) // 96            # rows of one tile lie more than 2^32 bytes apart
            buf = torch.empty((rows - 1) * pitch + nc, dtype=torch.uint8, device="cuda")
            buf.as_strided((rows, nc), (pitch, 1)).copy_(op.macro.codes)
            scale = _Strided(buf, pitch, 1, 0)
            scale.first = 0
        return scale

    want, got = (torch.empty(m, n, dtype=torch.float32, device="cuda") for _ in range(2))
    L.gemm_mxfp4_two_level(m, n, k, a.codes, a.scales, a.macro, b.codes, b.scales, b.macro, want)
    L.gemm_mxfp4_two_level(m, n, k, a.codes, a.scales, moved(a), b.codes, b.scales, moved(b), got)
    assert torch.equal(got, want)


def test_tensors_of_another_device_are_not_handed_to_a_launch_here(monkeypatch):
    """The two helpers also serve tensors of a device that is not current, as tensor operations do."""
    from alto_b200.grouped import group_experts_from_offsets
    offs = torch.tensor([128, 384], dtype=torch.int32, device="cuda")
    scales = torch.randint(1, 255, (96, 6), dtype=torch.uint8, device="cuda")
    experts, packed = group_experts_from_offsets(offs, 600), E.pack_plain_scales(scales, 96, False, 32)

    def launched(*args, **kw):
        raise AssertionError("a launch on the current device")

    other = torch.cuda.current_device() + 1
    monkeypatch.setattr(torch.cuda, "current_device", lambda: other)
    monkeypatch.setattr(L, "group_experts", launched)
    monkeypatch.setattr(L, "pack_scales", launched)
    assert torch.equal(group_experts_from_offsets(offs, 600), experts)
    assert torch.equal(E.pack_plain_scales(scales, 96, False, 32), packed)
