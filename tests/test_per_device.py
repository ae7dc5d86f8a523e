"""Set-up kept per device (csrc/per_device.cuh): once on each device, again after a failure, thread-safe."""

import shutil
import subprocess

import pytest

from conftest import REPO

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.cuh"
int main() {
  cphf::PerDevice p;
  std::atomic<int> calls[3] = {};
  auto set = [&](int d) { return p.once(d, [&] { ++calls[d]; return true; }); };
  std::vector<std::thread> ts;
  for (int i = 0; i < 16; ++i) ts.emplace_back([&, i] { for (int k = 0; k < 100; ++k) if (!set(i % 2)) ++calls[2]; });
  for (auto& t : ts) t.join();
  int tries = 0;
  const bool first = p.once(5, [&] { return ++tries > 1; }), second = p.once(5, [&] { return ++tries > 1; });
  const bool third = p.once(5, [&] { return ++tries > 1; });
  int far = 0;  // devices beyond the table are set up at each call
  for (int k = 0; k < 3; ++k) p.once(99, [&] { ++far; return true; });
  std::printf("%d %d %d %d %d %d %d %d\n", calls[0].load(), calls[1].load(), calls[2].load(), first, second, third, tries, far);
}
"""


def test_each_device_is_set_up_once(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-pthread", "-I", str(REPO / "rstsr-showcase-hessian_gb300" / "csrc"), str(src),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["1", "1", "0", "0", "1", "1", "2", "3"]
