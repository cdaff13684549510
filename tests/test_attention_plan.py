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
  if (!std::strcmp(argv[1], "cluster")) return std::printf("%d\n", decode_cluster_size(n(2), n(3), 148)), 0;
  const Units u{n(2), 128 / n(3), (n(2) + 128 / n(3) * 2 - 1) / (128 / n(3) * 2), 0, n(4) / 64};  // Q, G, block size
  if (!std::strcmp(argv[1], "row_cost")) std::printf("%lld\n", row_cost(u, n(5)));
  if (!std::strcmp(argv[1], "may_be_cut")) std::printf("%d\n", may_be_cut(u, n(6), n(5), n(7), 148));
  if (!std::strcmp(argv[1], "cut")) {  // rows whose counts follow
    long long total = 0;
    int lo = 1 << 30, hi = 0, nc;
    for (int i = 5; i < argc; ++i) {
      total += row_cost(u, n(i));
      if (n(i) < lo) lo = n(i);
      if (n(i) > hi) hi = n(i);
    }
    std::printf("%d\n", units_are_cut(total, static_cast<long long>(argc - 5) * u.n_pairs, unit_cost(u, lo, 0), unit_cost(u, hi, u.n_pairs - 1), 148, &nc));
  }
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


@pytest.mark.parametrize("rows", [1, 2, 8, 37, 72, 148, 150])
@pytest.mark.parametrize("Q,G", [(64, 4), (700, 7), (1152, 4), (2048, 8)])
@pytest.mark.parametrize("cap", [0, 20, 64, 300])
def test_dense_launches_merge_where_units_are_cut(plan, rows, Q, G, cap):
    assert plan("may_be_cut", Q, G, 64, cap, rows, 1) == plan("cut", Q, G, 64, *[cap] * rows)


def test_table_launches_merge_where_units_may_be_cut(plan):
    assert plan("may_be_cut", 128, 4, 64, 62, 72, 0) == 0   # 144 units of at most 32 steps on 148 CTAs: as before they stay whole
    assert plan("may_be_cut", 128, 4, 64, 200, 72, 0) == 1  # ... of up to 101 steps: a row may be worth cutting
    assert plan("may_be_cut", 128, 4, 64, 62, 20, 0) == 1   # 40 units: most CTAs would idle
    assert plan("may_be_cut", 128, 4, 64, 10, 20, 0) == 0   # at most six steps: nothing to gain
    # whatever the counts, what may not be cut is dealt out whole by the kernel's own rule or was excluded above
    for counts in ([10] * 20, [0] * 19 + [10], list(range(11)) * 2):
        assert plan("cut", 128, 4, 64, *counts) == 0


@pytest.mark.parametrize("rows,subs,want", [
    (1, 1, 1), (1, 3, 1), (1, 4, 2), (8, 16, 8), (32, 512, 8),
    (33, 512, 4), (36, 512, 4), (37, 512, 4),  # as clusters of 8 they would take two waves
    (64, 128, 4), (65, 128, 2), (74, 128, 2), (148, 128, 2), (150, 128, 1), (296, 128, 1),
    (297, 128, 2), (304, 128, 2), (400, 128, 2), (304, 8, 1), (1024, 2048, 2), (1024, 1, 1),
])
def test_decode_cluster_size(plan, rows, subs, want):
    cs = plan("cluster", rows, subs)
    waves = {c: -(-rows * c // (296 if c < 4 else 259)) for c in (1, 2, 4, 8) if (c == 1 or subs >= 2 * c) and (c < 8 or rows * 8 <= 259)}
    cost = {c: w * (subs / c + 16) for c, w in waves.items()}
    assert cost[cs] == min(cost.values())
    assert cs == want
