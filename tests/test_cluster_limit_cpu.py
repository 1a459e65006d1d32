"""The number of resident clusters is asked once per device; a question that fails is put again and leaves no error behind: the header
against stand-ins for the runtime calls it makes."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
INCLUDE = "/usr/local/cuda/include"

PROGRAM = r"""
#include "common/cluster_limit.h"
#include <cstdio>
static int device = 0, fail_raise = 0, fail_ask = 0, asked = 0;
static cudaError_t left = cudaSuccess;
static cudaError_t leave(cudaError_t e) { if (e != cudaSuccess) left = e; return e; }
extern "C" cudaError_t CUDARTAPI cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t CUDARTAPI cudaGetLastError() { const cudaError_t e = left; left = cudaSuccess; return e; }
extern "C" cudaError_t CUDARTAPI cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) {
  return leave(fail_raise ? cudaErrorInvalidValue : cudaSuccess);
}
extern "C" cudaError_t CUDARTAPI cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) {
  ++asked;
  *n = fail_ask ? 99 : 70 + device;
  return leave(fail_ask ? cudaErrorUnknown : cudaSuccess);
}
int main() {
  static dptb::SmemLimit smem;
  static dptb::ClusterLimit limit;
  const int k = 1;
  cudaLaunchConfig_t cfg = {};
  auto ask = [&] { std::printf("%d:%d ", limit.resident(&k, smem, 100, cfg), (int)left); };
  fail_raise = 1; ask(); fail_raise = 0;
  fail_ask = 1; ask(); fail_ask = 0;
  for (int d : {0, 0, 1, 0, 63, 64, 64}) { device = d; ask(); }
  std::printf("%d\n", asked);
}
"""


@pytest.mark.skipif(not shutil.which("g++") or not os.path.isdir(INCLUDE), reason="no host compiler or CUDA headers")
def test_questions(tmp_path):
    src, exe = tmp_path / "limit.cpp", tmp_path / "limit"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", f"-I{ROOT}/csrc", f"-I{INCLUDE}", str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["0:0", "0:0", "70:0", "70:0", "71:0", "70:0", "133:0", "134:0", "134:0", "6"]


def test_nobody_asks_without_it():
    for folder, _, files in os.walk(os.path.join(ROOT, "csrc")):
        for name in files:
            with open(os.path.join(folder, name)) as f:
                assert name == "cluster_limit.h" or "cudaOccupancyMaxActiveClusters" not in f.read(), name
