"""A kernel's launch settings, on the CPU with a fake of the two runtime calls: made on every device that
launches it, once each; a setting that failed is tried again. And no launcher sets them another way."""
import re
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "shaderous_b200" / "csrc"

PROGRAM = r"""
#include "launch_attr.h"
#include <cstdio>
static int current = 0, fail_next = 0, sets[80][2];
extern "C" cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute a, int) {
  if (fail_next) { fail_next = 0; return cudaErrorInvalidValue; }
  sets[current][a == cudaFuncAttributePreferredSharedMemoryCarveout]++;
  return cudaSuccess;
}
#define WANT(x) if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; }
int main() {
  static shz::LaunchAttr attr, plain;
  const int k = 0;
  for (int turn = 0; turn < 3; turn++)
    for (int dev : {0, 1, 63}) {
      current = dev;
      WANT(attr.set(&k, 108 << 10, true) == cudaSuccess);
      WANT(sets[dev][0] == 1 && sets[dev][1] == 1);
    }
  current = 70;  // beyond what is kept: every launch
  for (int n = 1; n <= 2; n++) WANT(attr.set(&k, 108 << 10, true) == cudaSuccess && sets[70][0] == n);
  current = 2;
  fail_next = 1;
  WANT(plain.set(&k, 60 << 10, false) == cudaErrorInvalidValue && sets[2][0] == 0);
  for (int n = 0; n < 2; n++) WANT(plain.set(&k, 60 << 10, false) == cudaSuccess && sets[2][0] == 1 && sets[2][1] == 0);
  return 0;
}
"""


def test_settings_are_made_once_on_each_device(tmp_path):
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), "-I", "/usr/local/cuda/include", str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_every_launcher_sets_them_so():
    users = [p.name for p in CSRC.iterdir() if p.suffix in (".cu", ".cuh", ".h", ".cpp")
             and re.search(r"cudaFuncSetAttribute\s*\(", p.read_text())]
    assert users == ["launch_attr.h"]
