"""Launch limits and kernel attributes are found once per device, not once per process
(PerDevice in benchmarks_gb300/csrc/mfgb_internal.h), run on the host with device numbers."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include <cstdio>
#include <thread>
#include "mfgb_internal.h"
int main() {
  static mfgb::PerDevice found;
  int calls[66] = {};
  for (int round = 0; round < 3; ++round)
    for (int dev : {0, 3, 63, 64, -1})
      if (found.get(dev, [&] { ++calls[dev + 1]; return 10 + dev; }) != 10 + dev) return 1;
  if (calls[1] != 1 || calls[4] != 1 || calls[64] != 1) return 2;  // once each
  if (calls[65] != 3 || calls[0] != 3) return 3;                   // no such slot: every time
  if (found.get(7, [] { return 0; }) != 0 || found.get(7, [] { return 5; }) != 0) return 4;
  std::thread t[8];
  std::atomic<int> bad{0};
  for (auto &x : t) x = std::thread([&] { bad += found.get(9, [] { return 42; }) != 42; });
  for (auto &x : t) x.join();
  return bad ? 5 : 0;
}
"""


def test_found_once_per_device(tmp_path):
    from benchmarks_gb300 import build
    src, exe = tmp_path / "d.cu", tmp_path / "d"
    src.write_text(PROGRAM)
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-I" + build.CSRC,
                    "-I" + os.path.join(ROOT, "include"), str(src), "-o", str(exe)], check=True, timeout=300)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0
