"""The drain of a TMA ring after an expired wait (``csrc/ca_ring.cuh``), on the CPU: against a model of the ring in which
every entry's copies are counted, the last ``stages`` issued ones are still in flight, and the next is never issued."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "compactattention_b200" / "csrc"

SOURCE = r"""
#include <cstdio>
#include <vector>
#include "ca_ring.cuh"

int main() {
  for (int stages = 1; stages <= 5; ++stages) {
    for (int issued = 0; issued <= 4 * stages + 1; ++issued) {
      // entry e uses stage e % stages for the (e / stages)-th time and completes that stage's phase of that number
      std::vector<int> in_flight(issued, 0);
      for (int e = issued > stages ? issued - stages : 0; e < issued; ++e) in_flight[e] = 1;
      bool wrong = false;
      ca::drain_ring(issued, stages, [&](int stage, unsigned parity) {
        bool found = false;
        for (int e = 0; e < issued; ++e) {
          if (in_flight[e] && e % stages == stage && ((e / stages) & 1) == static_cast<int>(parity)) in_flight[e] = 0, found = true;
        }
        wrong |= !found;  // waits for a phase that nothing will complete, or that is over
      });
      for (int e = 0; e < issued; ++e) wrong |= in_flight[e] != 0;
      if (wrong) return std::printf("stages %d issued %d\n", stages, issued), 1;
    }
  }
  return 0;
}
"""


def test_every_issued_copy_is_waited_for(tmp_path):
    (tmp_path / "ring.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", f"-I{CSRC}", "-o", str(tmp_path / "ring"), str(tmp_path / "ring.cpp")], check=True)
    out = subprocess.run([str(tmp_path / "ring")], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


def test_only_issued_entries_are_counted():
    """The decode kernel counts an entry after its copies, and drains whichever role's wait expired."""
    text = (CSRC / "ca_attn_decode.cu").read_text()
    loads, count = text.rindex("tma_load_4d("), text.index("++issued;")
    assert text.count("++issued") == 1 and loads < count < loads + 200
    assert "if (sh->abort_flag) give_up(" in text[text.rindex("cluster.sync();"):]
