"""Kernel attributes belong to the device that is current when they are set: they are set on each device once, and nowhere
once for the process."""
import os
import re
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "hdiscontinuousgalerkin.jl_gb300", "csrc")

_PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <stdexcept>
#include <thread>
#include <vector>
#include "once_per_device.h"
int main() {
  OncePerDevice once;
  std::atomic<int> calls[80] = {};
  try {
    once(3, [] { throw std::runtime_error("not yet"); });
    return 1;
  } catch (const std::runtime_error&) {
  }
  std::vector<std::thread> ts;
  for (int t = 0; t < 8; ++t)
    ts.emplace_back([&] {
      for (int k = 0; k < 160; ++k) once(k % 80, [&] { ++calls[k % 80]; });
    });
  for (auto& t : ts) t.join();
  for (int d = 0; d < 80; ++d)
    if (calls[d] != 1) return 2;
  std::puts("ok");
  return 0;
}
"""


def test_each_device_once(tmp_path):
    (tmp_path / "t.cpp").write_text(_PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", CSRC, "-o", str(tmp_path / "t"), str(tmp_path / "t.cpp")],
                   check=True)
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok"


def test_no_attribute_is_set_once_for_the_process():
    """Every cudaFuncSetAttribute is guarded per device, or not at all."""
    for name in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, name)).read()
        if "cudaFuncSetAttribute" not in text:
            continue
        assert "call_once" not in text and "once_flag" not in text, name
        for m in re.finditer(r"static\s+(?:std::atomic<)?bool>?\s+(\w+)[^;]*;\s*if\s*\(!\1\b", text):
            assert "cudaFuncSetAttribute" not in text[m.end():m.end() + 300], (name, m.group(0))
