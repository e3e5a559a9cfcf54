"""Kernel attributes belong to a device: what is set once is set once per device, and no launcher
remembers it in a flag of the whole process."""
import glob
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "graft.jl_gb300", "csrc")

PROGRAM = r"""
#include "gtn_once.h"
#include <cstdio>
int main() {
  PerDeviceOnce once;
  int calls[70] = {};
  auto set = [&](int dev, int result) { return once(dev, [&] { ++calls[dev]; return result; }); };
  bool ok = set(0, 0) == 0 && set(0, 0) == 0 && calls[0] == 1;      // once on device 0
  ok = ok && set(1, 0) == 0 && set(1, 0) == 0 && calls[1] == 1;     // and once on device 1
  ok = ok && set(5, 3) == 3 && set(5, 0) == 0 && set(5, 0) == 0 && calls[5] == 2;  // again after a failure
  ok = ok && set(63, 0) == 0 && set(63, 0) == 0 && calls[63] == 1;
  ok = ok && set(64, 0) == 0 && set(64, 0) == 0 && calls[64] == 2;  // beyond the mask: every time
  return ok ? 0 : 1;
}
"""


def test_once_per_device(tmp_path):
    src = tmp_path / "once.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "once"
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    subprocess.run([str(exe)], check=True)


def test_launchers_keep_no_flag_of_the_process():
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        text = open(path).read()
        assert "cudaFuncSetAttribute" not in text, path  # func_attribute and smem_opt_in call it
        assert not re.search(r"static bool attr", text), path
