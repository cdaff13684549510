"""Contracts of the kernels that their sources show and no run can be relied on to break: a wait without a reader of its result
goes on to touch what it waited for; a load through the non-coherent path promises that nobody writes the address while the kernel
lives, which a programmatic dependent launch cannot promise of what the launch before it writes."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "compactattention_b200" / "csrc"


def _without_comments(path):
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", path.read_text(), flags=re.S))


def test_no_wait_result_is_dropped():
    """Only the drains after an abort (their flag is a dummy) may ignore how their wait ended."""
    seen = 0
    for path in sorted(CSRC.glob("*.cu")):
        text = _without_comments(path)
        for call in re.finditer(r"ptx::mbar_wait_\w+\(", text):
            statement = text[call.start():text.index(";", call.start())]
            before = text[:call.start()].rstrip()[-1]
            seen += 1
            assert before not in "{};)" or "&dummy" in statement, f"{path.name}: {statement}"
    assert seen > 15


def test_the_self_test_runs_every_wait_routine():
    """``ca_selftest_bounded_wait`` lets each of them run out (a GPU test reads how that ended)."""
    routines = re.findall(r"\bbool (mbar_wait_\w+)\(", _without_comments(CSRC / "ca_common.cuh"))
    kernel = _without_comments(CSRC / "ca_runtime.cu").split("selftest_bounded_wait_kernel(", 1)[1].split("extern \"C\"")[0]
    assert len(routines) >= 2 and all(f"{name}(" in kernel for name in routines)


def test_dependent_launches_load_coherently():
    """Every kernel here may be resident while the launch before it still writes, and its pointers come as plain arguments, so
    only an ordinary load stays behind the dependency wait by contract."""
    for path in sorted(CSRC.glob("*.cu*")):
        text = _without_comments(path)
        found = re.findall(r"__ldg|ld\.global\.nc|const\s[^,;(){}]*\*\s*__restrict__", text)
        assert not found, f"{path.name}: {found}"


def test_the_self_tests_limit_covers_the_coarse_clock():
    """``mbar_wait_lean`` keeps time in units of 1024 ns with the lowest bit set.  For every start within a pair of units and short limit,
    the limit that the self-test passes may not let the wait end before ``limit_ns``."""
    kernel = _without_comments(CSRC / "ca_runtime.cu").split("selftest_bounded_wait_kernel(", 1)[1].split("extern \"C\"")[0]
    extra = int(re.search(r"\(limit_ns \+ 999\) / 1000\)(?: \+ (\d+))?\);", kernel).group(1) or 0)
    for limit_ns in (1, 500, 1000, 1024, 3000, 10_000, 40_000):
        limit = (limit_ns + 999) // 1000 + extra
        for start in range(0, 2048, 64):
            t0 = (start >> 10) | 1
            end = next(t for t in range(start, start + 10**6, 64) if ((t >> 10) | 1) - t0 > limit)
            assert end - start >= limit_ns, (limit_ns, start)
