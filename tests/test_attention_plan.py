"""The attention kernel's planning arithmetic (``csrc/ca_attn_plan.cuh``), compiled for the host."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "compactattention_b200" / "csrc"

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "ca_attn_plan.cuh"
using namespace ca::attn;

int main(int argc, char** argv) {
  auto n = [&](int i) { return std::atoi(argv[i]); };
  const Units u{n(2), 128 / n(3), (n(2) + 128 / n(3) * 2 - 1) / (128 / n(3) * 2), 0, n(4) / 64};  // Q, G, block size
  if (!std::strcmp(argv[1], "row_cost")) std::printf("%lld\n", row_cost(u, n(5)));
  return 0;
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-ftrapv", "-Wall", "-Werror", f"-I{CSRC}", "-o", str(d / "plan"), str(d / "plan.cpp")], check=True)
    return lambda *a: int(subprocess.run([str(d / "plan"), *map(str, a)], check=True, capture_output=True, text=True).stdout)


@pytest.mark.parametrize("Q,G,bs,count", [
    (1, 1, 64, 0), (64, 4, 64, 7), (1000, 7, 128, 33), (8192, 4, 64, 0),
    (1 << 20, 128, 64, 0),       # a first chunk of a million tokens, 128 heads to the KV head: 2^31 steps
    (1 << 19, 128, 64, 1 << 14),  # and half a million behind a million
])
def test_a_rows_cost_is_the_sum_of_its_units(plan, Q, G, bs, count):
    tokens = 2 * (128 // G)  # of a unit
    want = 0
    for t in range(0, Q, tokens):
        subs = count * (bs // 64) + (min(t + tokens, Q) - 1) // 64 + 1
        want += (subs + 1) // 2 + 3
    assert plan("row_cost", Q, G, bs, count) == want
