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
