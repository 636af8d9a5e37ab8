"""The opt-in to large dynamic shared memory is kept per kernel and device: compiled against a
stand-in of the two runtime calls, it is made once on every device (a failed one again), and
no kernel of the library has an opt-in of another kind."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "msbg_gb300", "csrc")
MAIN = r"""
#include "smem_optin.h"
static int device, calls, failing;
extern "C" cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute a, int bytes) {
  if (a != cudaFuncAttributeMaxDynamicSharedMemorySize || bytes != 100000) return cudaErrorInvalidValue;
  calls++;
  return failing ? cudaErrorInvalidDevice : cudaSuccess;
}
int main() {
  static msbg::SmemOptIn first, second;
  for (int round = 0; round < 3; round++)
    for (device = 0; device < 8; device++)
      if (first(nullptr, 100000) != cudaSuccess) return 1;
  if (calls != 8) return 2;
  device = 3;
  if (second(nullptr, 100000) != cudaSuccess || calls != 9) return 3;  // another kernel
  device = 9;
  failing = 1;
  if (first(nullptr, 100000) == cudaSuccess || calls != 10) return 4;
  failing = 0;
  if (first(nullptr, 100000) != cudaSuccess || first(nullptr, 100000) != cudaSuccess || calls != 11) return 5;
  device = 100;  // beyond the mask: set on every call
  for (int k = 0; k < 2; k++)
    if (first(nullptr, 100000) != cudaSuccess) return 6;
  return calls == 13 ? 0 : 7;
}
"""


def _cuda_include():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    return os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")


def test_opt_in_once_per_kernel_and_device(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    src, exe = tmp_path / "optin.cpp", tmp_path / "optin"
    src.write_text(MAIN)
    r = subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-Werror", "-I", CSRC, "-isystem", _cuda_include(),
                        str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert subprocess.run([str(exe)]).returncode == 0


def test_every_opt_in_goes_through_it():
    for name in sorted(os.listdir(CSRC)):
        if name != "smem_optin.h":
            with open(os.path.join(CSRC, name)) as f:
                assert "cudaFuncSetAttribute" not in f.read(), name
