"""Launchers set a kernel's attributes once per device: a second device of the
same process must be set too (before, only the first one was, and a kernel with
more than 48 KB of dynamic shared memory could not launch on another).  The
helper is plain C++ and is compiled and run here."""
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bonzo_b200", "csrc")

SRC = r"""
#include "bnz_per_device.h"
#include <cstdio>
#include <thread>
#include <vector>
int main() {
  static PerDevice once;
  int made[66] = {0};
  for (int round = 0; round < 3; ++round)
    for (int dev = -1; dev < 65; ++dev) {
      const int x = once.get(dev, [&] { ++made[dev + 1]; return dev + 100; });
      if (x != dev + 100) return 1;
    }
  for (int dev = 0; dev < 64; ++dev)
    if (made[dev + 1] != 1) return 2;
  if (made[0] != 3 || made[65] != 3) return 3;  // a device it cannot hold is asked every time
  static PerDevice shared;
  std::vector<std::thread> t;
  std::atomic<int> bad{0};
  for (int q = 0; q < 8; ++q)
    t.emplace_back([&] {
      for (int n = 0; n < 10000; ++n)
        if (shared.get(n % 4, [&] { return n % 4 + 1; }) != n % 4 + 1) ++bad;
    });
  for (auto& x : t) x.join();
  return bad ? 4 : 0;
}
"""


def test_per_device(tmp_path):
    (tmp_path / "t.cpp").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-I", CSRC, str(tmp_path / "t.cpp"), "-o",
                    str(tmp_path / "t")], check=True)
    assert subprocess.run([str(tmp_path / "t")]).returncode == 0


def test_launchers_keep_nothing_for_the_first_device_only():
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh", ".h")):
            src = open(os.path.join(CSRC, f)).read()
            for m in re.finditer(r"FuncSetAttribute|MaxActiveBlocks", src):
                before = src[:m.start()].rsplit("\n}\n", 1)[-1]  # the function it stands in
                assert not re.search(r"static (int|bool) ", before), (f, before[-300:])
