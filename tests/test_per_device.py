"""Launch limits are asked of each device once (axicor_gb300/csrc/per_device.h), on the CPU with devices that differ."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "axicor_gb300" / "csrc"

PROBE = r"""
#include <cstdio>
#include <initializer_list>
#include "per_device.h"
int main() {
  static axc::PerDevice<unsigned> sms;
  int made = 0;
  auto ask = [&](int dev) { return sms.get(dev, [&] { made++; return 100u + (unsigned)dev; }); };
  for (int round = 0; round < 2; round++)
    for (int dev : {0, 3, 1, 63}) printf("%u ", ask(dev));
  printf("%d ", made);
  printf("%u ", ask(-1));
  printf("%u ", ask(64));
  printf("%d\n", made);
}
"""


def test_each_device_has_its_own_answer(tmp_path):
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(PROBE)
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert out[:8] == ["100", "103", "101", "163"] * 2
    assert out[8] == "4", "once a device"
    assert out[9:] == ["99", "164", "6"], "beyond the table: asked each time"

