"""The once-per-device helper of the kernel launches (csrc/device_once.h), built with the host
compiler: two devices in one process, several threads, an exception.  (Two devices themselves need
a second GPU.)"""
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "mpskit.jl_gb300", "csrc")

PROGRAM = r"""
#include "device_once.h"
#include <atomic>
#include <stdexcept>
#include <thread>
#include <vector>
int main() {
  static gb::DeviceOnce once;
  std::atomic<int> n[3] = {};
  std::vector<std::thread> t;
  for (int i = 0; i < 12; ++i)
    t.emplace_back([&, i] {
      for (int k = 0; k < 100; ++k) once(i % 3, [&] { ++n[i % 3]; });
    });
  for (auto& x : t) x.join();
  for (auto& c : n)
    if (c != 1) return 1;
  static gb::DeviceOnce again;
  int tries = 0;
  for (int k = 0; k < 3; ++k) {
    try {
      again(5, [&] { if (++tries == 1) throw std::runtime_error("first"); });
    } catch (const std::runtime_error&) {
      if (k != 0) return 2;
    }
  }
  if (tries != 2) return 3;
  int far = 0;
  again(1000, [&] { ++far; });
  again(1000, [&] { ++far; });
  return far == 2 ? 0 : 4;
}
"""


def test_once_per_device(tmp_path):
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(src), "-o", str(exe)],
                   check=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0


def test_kernel_attributes_are_set_per_device():
    """Every cudaFuncSetAttribute stands under a DeviceOnce, none under a flag of the process."""
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        text = open(os.path.join(CSRC, name)).read()
        for m in re.finditer(r"cudaFuncSetAttribute", text):
            before = text[:m.start()]
            at = max(before.rfind("static DeviceOnce"), before.rfind("static std::once_flag"))
            assert at >= 0 and before[at:].startswith("static DeviceOnce"), (name, before[-200:])
