"""Launch configurations are kept per device (csrc/perdevice.cuh): host code, with
made-up device numbers."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "isai_kernel_gb300", "csrc")

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "perdevice.cuh"

int main() {
  bilu::PerDevice<int> c;
  std::atomic<int> made{0}, wrong{0};
  std::vector<std::thread> ts;
  for (int t = 0; t < 16; ++t)
    ts.emplace_back([&, t] {
      for (int i = 0; i < 1000; ++i) {
        const int dev = (t + i) % 3;
        int v = -1;
        const int rc = c.get(dev, &v, [&](int* p) { ++made; *p = 100 + dev; return 0; });
        if (rc != 0 || v != 100 + dev) ++wrong;
      }
    });
  for (auto& t : ts) t.join();
  // a device whose first call fails is asked again
  int v = -1, calls = 0;
  auto fails_once = [&](int* p) { *p = 7; return calls++ == 0 ? -5 : 0; };
  const int a = c.get(9, &v, fails_once), kept = v, b = c.get(9, &v, fails_once);
  std::printf("%d %d %d %d %d %d\n", made.load(), wrong.load(), a, kept, b, v);
}
"""


def test_a_value_per_device(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    src = tmp_path / "per_device.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "per_device"
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(src), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout
    assert out.split() == ["3", "0", "-5", "-1", "0", "7"]


def test_no_launch_configuration_of_the_first_device():
    """No function keeps a grid, an SM count or a kernel attribute in a plain static."""
    import re

    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            text = open(os.path.join(CSRC, name)).read()
            assert not re.search(r"^\s+static (int|bool|size_t) \w+ = ", text, re.M), name
