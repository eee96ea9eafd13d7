"""Every form of the bounded wait, complete, run into its limit and called off by another role, at several limits."""
import pytest

pytestmark = pytest.mark.gpu

from alto_b200 import _lib as L


@pytest.mark.parametrize("limit_ns", [300_000, 1_000_000, 30_000_000])
def test_waits_end_and_are_reported_once(limit_ns):
    assert L.status_read()[0] == 0
    L.selftest_wait_timeout(limit_ns)
    st, detail = L.status_read()
    assert st == L.E_TIMEOUT and detail == [9, 0, 99, 0]      # (100 and more: the first wait that was not as it should be)
    assert L.status_read() == (0, [0, 0, 0, 0])
