"""Work done once per device (kernels' shared-memory limits): every device of a
process gets it, a failed try is repeated, and threads do not repeat it. Host
code, compiled and run here."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <stdexcept>
#include <thread>
#include "hd_device_once.h"
int main() {
  static hd::OncePerDevice once, other;
  std::atomic<int> n[8] = {};
  for (int round = 0; round < 2; ++round)
    for (int d : {1, 0, 7, 1}) once.run(d, [&] { ++n[d]; });
  for (int d = 0; d < 8; ++d)
    if (n[d] != (d == 0 || d == 1 || d == 7)) return 1;
  other.run(1, [&] { ++n[1]; });  // each use has its own
  if (n[1] != 2) return 2;
  int tries = 0;
  for (int k = 0; k < 3; ++k) try {
    other.run(3, [&] { if (++tries == 1) throw std::runtime_error("x"); });
  } catch (const std::exception &) {}
  if (tries != 2) return 3;
  std::thread th[4];
  for (auto &t : th) t = std::thread([&] { for (int d = 0; d < 8; ++d) other.run(d, [&] { ++n[d]; }); });
  for (auto &t : th) t.join();
  return n[5] == 1 && n[6] == 1 && n[3] == 0 ? 0 : 4;
}
"""


def test_once_per_device(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "hammingdist_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0
