"""per_device.h: what a launch site forms once on each device (kernel attributes hold
for one device of a process) is formed on every ordinal, once, with its own result."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "curvib_old_gb300" / "csrc"

MAIN = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.h"
int main() {
  cvb::PerDevice p;
  int formed[80] = {};
  auto ask = [&](int dev, bool r) { return p.get(dev, [&] { formed[dev]++; return r; }); };
  for (int round = 0; round < 3; round++)
    for (int dev = 0; dev < 80; dev++)
      if (ask(dev, dev % 3 != 1) != (dev % 3 != 1)) return std::printf("result of %d\n", dev), 1;
  for (int dev = 0; dev < 64; dev++)
    if (formed[dev] != 1) return std::printf("formed %d times on %d\n", formed[dev], dev), 1;
  for (int dev = 64; dev < 80; dev++)
    if (formed[dev] != 3) return std::printf("formed %d times on %d\n", formed[dev], dev), 1;
  if (!p.get(-1, [] { return true; })) return 1;
  cvb::PerDevice q;  // threads on devices of their own
  std::atomic<int> wrong{0};
  std::vector<std::thread> ts;
  for (int dev = 0; dev < 8; dev++)
    ts.emplace_back([&, dev] {
      for (int k = 0; k < 1000; k++)
        if (q.get(dev, [&] { return dev % 2 == 0; }) != (dev % 2 == 0)) wrong++;
    });
  for (auto &t : ts) t.join();
  return wrong != 0;
}
"""


def test_once_on_each_device(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    (tmp_path / "main.cpp").write_text(MAIN)
    subprocess.run([cxx, "-std=c++17", "-pthread", "-I", str(CSRC), str(tmp_path / "main.cpp"), "-o",
                    str(tmp_path / "main")], check=True)
    r = subprocess.run([str(tmp_path / "main")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_no_attribute_once_a_process():
    """Every launch site that sets a kernel attribute does so through PerDevice."""
    for f in sorted(CSRC.glob("*.cu")):
        text = f.read_text()
        assert "static bool attr" not in text, f.name
        assert "cudaFuncSetAttribute" not in text or f.name == "kernels_tail.cu", f.name
