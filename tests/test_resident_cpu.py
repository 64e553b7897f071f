"""CPU test of the per-device memory of a kernel's resident CTAs (runtime.h): compiled with a device of its own."""
import pathlib
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include <cstdio>
#include "runtime.h"
namespace accgb {
static Device g;
const Device &device_info() { return g; }
}  // namespace accgb
using namespace accgb;
int main() {
  static ResidentCache cache{};
  int asked = 0, bad = 0;
  auto on = [&](int dev, int answer) {
    g.id = dev;
    return resident_once(cache, [&] { ++asked; return answer; });
  };
  bad += on(0, 3) != 3 || asked != 1;    // the first question on a device
  bad += on(0, 9) != 3 || asked != 1;    // remembered there
  bad += on(1, 2) != 2 || asked != 2;    // another device has its own
  bad += on(0, 9) != 3 || on(1, 9) != 2 || asked != 2;
  bad += on(5, 0) != 0 || on(5, -1) != 0 || asked != 4;  // a failed question is asked again
  bad += on(5, 4) != 4 || on(5, 9) != 4 || asked != 5;
  bad += on(64, 6) != 6 || on(64, 7) != 7 || on(-1, 8) != 8 || asked != 8;  // past the table: never kept
  std::printf("%d failed\n", bad);
  return bad != 0;
}
"""


def test_resident_ctas_are_remembered_per_device(tmp_path):
    cxx, cuda = shutil.which("g++"), pathlib.Path("/usr/local/cuda/include")
    if cxx is None or not (cuda / "cuda_runtime.h").exists():
        pytest.skip("no C++ compiler or CUDA headers")
    src, exe = tmp_path / "resident.cpp", tmp_path / "resident"
    src.write_text(PROGRAM)
    cmd = [cxx, "-std=c++17", f"-I{ROOT / 'accelerate-llvm_gb300' / 'csrc'}", f"-I{cuda}", str(src), "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
