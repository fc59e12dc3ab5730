"""Kernel attributes are set once per device, not once per process: hm_per_device.h against a CUDA
runtime of two devices made here, compiled for the host."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RUNTIME = """
#pragma once
enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1 };
inline int g_device = 0;
inline cudaError_t g_status = cudaSuccess;
inline cudaError_t cudaGetDevice(int *d) { *d = g_device; return g_status; }
"""

MAIN = """
#include "hm_per_device.h"
#include <cstdio>
int calls[100];
cudaError_t result = cudaSuccess;
template <int K> cudaError_t attrs() {
  static hm::PerDevice once;
  return once([] { calls[g_device] += K; return result; });
}
#define CHECK(c) if (!(c)) { std::printf("line %d\\n", __LINE__); return 1; }
int main() {
  CHECK(attrs<1>() == cudaSuccess && attrs<1>() == cudaSuccess && calls[0] == 1);
  g_device = 1;  // the second device of the process
  CHECK(attrs<1>() == cudaSuccess && attrs<1>() == cudaSuccess && calls[1] == 1);
  g_device = 0;
  CHECK(attrs<1>() == cudaSuccess && calls[0] == 1);
  CHECK(attrs<10>() == cudaSuccess && calls[0] == 11);  // each kernel its own
  g_device = 63;
  result = cudaErrorInvalidValue;  // a failure is returned and tried again
  CHECK(attrs<1>() == cudaErrorInvalidValue && calls[63] == 1);
  result = cudaSuccess;
  CHECK(attrs<1>() == cudaSuccess && attrs<1>() == cudaSuccess && calls[63] == 2);
  g_device = 70;  // past the record: every time
  CHECK(attrs<1>() == cudaSuccess && attrs<1>() == cudaSuccess && calls[70] == 2);
  g_status = cudaErrorInvalidValue;
  CHECK(attrs<1>() == cudaErrorInvalidValue);
  return 0;
}
"""


def test_attributes_once_per_device(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "main"
    subprocess.run(["g++", "-std=c++17", "-I", str(tmp_path), "-I", os.path.join(REPO, "hmatrixgpu.jl_gb300", "csrc"),
                    str(tmp_path / "main.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
