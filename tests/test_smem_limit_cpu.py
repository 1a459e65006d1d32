"""Raised shared-memory limits are remembered per device: the header against stand-ins for the two runtime calls it makes."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
INCLUDE = "/usr/local/cuda/include"

PROGRAM = r"""
#include "common/smem_limit.h"
#include <cstdio>
static int device = 0, fail = 0;
extern "C" cudaError_t CUDARTAPI cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t CUDARTAPI cudaFuncSetAttribute(const void* k, cudaFuncAttribute, int bytes) {
  if (fail) return cudaErrorInvalidValue;
  std::printf("%d:%d:%d ", device, *static_cast<const int*>(k), bytes);
  return cudaSuccess;
}
int main() {
  static dptb::SmemLimit a, b;
  const int ka = 1, kb = 2;
  for (int d : {0, 0, 1, 1, 0, 63, 64, 64}) {
    device = d;
    if (a.raise(&ka, 100) != cudaSuccess) return 1;
  }
  device = 1;
  fail = 1;
  if (b.raise(&kb, 200) == cudaSuccess) return 2;
  fail = 0;
  if (b.raise(&kb, 200) != cudaSuccess || b.raise(&kb, 200) != cudaSuccess) return 3;
}
"""


@pytest.mark.skipif(not shutil.which("g++") or not os.path.isdir(INCLUDE), reason="no host compiler or CUDA headers")
def test_every_device_is_raised_once(tmp_path):
    src, exe = tmp_path / "limit.cpp", tmp_path / "limit"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", f"-I{ROOT}/csrc", f"-I{INCLUDE}", str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["0:1:100", "1:1:100", "63:1:100", "64:1:100", "64:1:100", "1:2:200"]


def test_no_launcher_remembers_it_for_the_process():
    for folder, _, files in os.walk(os.path.join(ROOT, "csrc")):
        for name in files:
            with open(os.path.join(folder, name)) as f:
                for body in re.findall(r"\n  static (?:bool|int) \w+ = [^\n]*(?:\n  .*){1,6}", f.read()):
                    assert "cudaFuncSetAttribute" not in body, (name, body)
