"""altob200_linear_backward refuses what it cannot do before it launches anything."""
import ctypes as C

import pytest

from alto_b200 import _lib as L

_BUFFER = C.create_string_buffer(4096)
_AT = (C.addressof(_BUFFER) + 255) // 256 * 256


def _call(**fields):
    a = L.LinearBackwardArgs()
    a.M, a.K, a.N, a.ld, a.format, a.dtype, a.use_outer = 32, 32, 32, 32, L.FMT_NVFP4, L.DT_BF16, 1
    for name in ("dy", "xm_codes", "xm_scales", "wt_codes", "wt_scales", "xm_outer", "wt_outer", "dx", "dw", "scratch"):
        setattr(a, name, _AT)
    for name, value in fields.items():
        setattr(a, name, value)
    return L.lib().altob200_linear_backward(a, _AT, None)


@pytest.mark.parametrize("missing", [dict(wt_outer=None), dict(xm_outer=None), dict(dw=None, wt_outer=None), dict(dx=None, xm_outer=None),
                                     dict(scratch=None), dict(wt_codes=None), dict(xm_scales=None), dict(dy=None), dict(N=48)])
def test_missing_parts_are_refused(missing):
    assert _call(**missing) == L.E_SHAPE
