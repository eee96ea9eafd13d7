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


def test_every_wait_has_a_site_of_its_own():
    header = (CSRC.parent.parent / "include" / "altob200.h").read_text()
    listed = header[header.index("its wait sites are"):header.index("free scale slot 17") + 18]
    documented = sorted(int(n) for n in re.findall(r"\b\d+\b", listed))
    assert documented == [*range(1, 7), *range(11, 18), *range(21, 27)]
    reported = []
    for name in ("gemm_sm100.cu", "gemm_macro.cuh"):
        for line in re.findall(r"report_timeout\(abort_flag, (.*)", (CSRC / name).read_text()):
            reported += [int(n) for n in re.findall(r"(?:^|[?:] )(\d+)(?=[ ;)])", line)]
    assert sorted(reported) == documented
