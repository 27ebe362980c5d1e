"""csrc/kept.h, the occupancy figure that the row kernels ask the runtime for once: kept per device and
shared-memory size, and not at all when the runtime could not answer."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "shmtensor_b200" / "csrc"

PROGRAM = r"""
#include "kept.h"
#include <cassert>

int main() {
  static shmt::KeptOccupancy kept;
  int asked = 0, answer = 4;
  bool can = false;
  auto ask = [&](int* n) { ++asked; *n = answer; return can; };
  assert(kept.get(0, 512, ask) == 1 && asked == 1);   // no answer: one CTA, for this call
  can = true;
  assert(kept.get(0, 512, ask) == 4 && asked == 2);   // asked again
  assert(kept.get(0, 512, ask) == 4 && asked == 2);   // kept
  answer = 2;
  assert(kept.get(1, 512, ask) == 2 && asked == 3);   // another device is asked itself
  assert(kept.get(0, 512, ask) == 4 && asked == 3);   // and does not displace the first
  assert(kept.get(0, 0, ask) == 2 && asked == 4);     // other shared memory is another question
  assert(kept.get(0, 512, ask) == 2 && asked == 5);
  assert(kept.get(64, 512, ask) == 2 && kept.get(64, 512, ask) == 2 && asked == 7);  // beyond the table
  assert(kept.get(-1, 512, ask) == 2 && asked == 8);
  answer = 0;
  assert(kept.get(2, 512, ask) == 1 && kept.get(2, 512, ask) == 1 && asked == 10);   // no CTA fits: not kept
  return 0;
}
"""


def test_occupancy_is_kept_per_device_and_only_when_answered(tmp_path):
    src, exe = tmp_path / "kept.cc", tmp_path / "kept"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-UNDEBUG", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    subprocess.run([str(exe)], check=True)
