"""When the row copy is laid out anew (layout_decision, axicor_gb300/csrc/engine.h), on the CPU."""
import subprocess
from pathlib import Path

from axicor_gb300.build import CUDA_HOME

CSRC = Path(__file__).resolve().parents[1] / "axicor_gb300" / "csrc"

PROBE = r"""
#include <cstdio>
#include <cstring>
#include "engine.h"
// Ticks between layouts of an unsettled shard whose weights and lit axons stay as they are, over 6,400 ticks.
static void run(unsigned streak, bool index) {
  axc::ShardCtl c;
  std::memset(&c, 0, sizeof(c));
  c.slot_total = 1000;
  c.pfx_total = 900;
  c.lay_wait = 16;
  c.streak = streak;
  unsigned last = 0;
  for (unsigned t = 0; t < 6400; t += 50) {
    axc::layout_decision(&c, t == 0, 50, 0, index);
    if (c.lay_now && t) {
      printf("%u ", t - last);
      last = t;
    }
  }
  printf("end ");
}
int main() {
  run(0, false);
  run(40, false);
  run(0, true);
  run(40, true);
}
"""


def test_periodic_layout_after_the_learned_engine(tmp_path):
    """A batch or per-tick call cannot run the sparse form: ticks that the learned engine left as sparse do not keep
    it from the layout that an unsettled shard gets every 1,600 ticks."""
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(PROBE)
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), "-I", str(CUDA_HOME / "include"), str(src), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("end")
    plain, after_learned, quiet_index, sparse_index = (x.split() for x in out[:4])
    assert plain == ["1600"] * 3
    assert after_learned == plain
    assert quiet_index == plain
    assert sparse_index == [], "the sparse form's rows stay"
