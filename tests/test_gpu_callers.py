"""Calls at the edge of what the host functions take."""
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
