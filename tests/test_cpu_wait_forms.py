"""The self-test kernel exercises the bounded waits that the GEMM kernels use, not others."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "alto_b200" / "csrc"


def test_self_test_waits_as_the_kernels_do():
    text = (CSRC / "gemm_sm100.cu").read_text()
    start = text.index("wait_selftest_kernel(uint64_t limit_ns) {")
    end = text.index("\n}\n", start)
    call = re.compile(r"\b(mbar_\w*wait\w*|report_timeout)\(")
    used = set(call.findall(text[:start] + text[end:] + (CSRC / "gemm_macro.cuh").read_text()))
    assert used and set(call.findall(text[start:end])) == used
