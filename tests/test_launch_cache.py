"""The launches' cache (host code, compiled here): every configuration is asked
for once, however many there are, and a failed one is asked for again."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "orthoroute_b200" / "csrc"
PROGRAM = r"""
#include "launch_cache.cuh"
int main() {
  static char kernels[150];
  orsp::LaunchCache cache;
  int asked = 0, value = 0;
  for (int round = 0; round < 3; ++round)
    for (int k = 0; k < 150; ++k)
      for (int depth = 1; depth <= 6; ++depth)
        for (int device = 0; device < 2; ++device) {
          if (cache.get(&kernels[k], 288, 1000 * depth, device, &value, [&](int *v) { *v = k * depth + device; return ++asked, 0; }))
            return 1;
          if (value != k * depth + device) return 2;
        }
  if (asked != 150 * 6 * 2) return 3;
  int failed = 0;
  for (int round = 0; round < 2; ++round)
    if (cache.get(&kernels[0], 1, 1, 0, &value, [&](int *) { return ++failed, -7; }) != -7) return 4;
  return failed == 2 ? 0 : 5;
}
"""


def test_every_configuration_is_asked_for_once(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host compiler")
    src, exe = tmp_path / "cache.cpp", tmp_path / "cache"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", f"-I{CSRC}", str(src), "-o", str(exe), "-pthread"], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
