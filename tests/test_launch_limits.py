"""A kernel's dynamic shared-memory limit is one value per kernel and device, shared by every handle and thread.
kernel_residency (tp_launch.h) may only raise it: a launch that follows its own call must still fit after another
thread's call for a smaller scene came in between.  CPU test: the header compiled against a small stand-in for the
CUDA runtime, which records the limits."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RUNTIME = r"""
#pragma once
#include <map>
#include <utility>
typedef int cudaError_t;
constexpr int cudaSuccess = 0, cudaErrorInvalidValue = 1;
enum cudaFuncAttribute { cudaFuncAttributeMaxDynamicSharedMemorySize };
enum cudaDeviceAttr { cudaDevAttrMultiProcessorCount };
inline int device = 0;
inline std::map<std::pair<const void *, int>, int> limit;
inline cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
inline cudaError_t cudaFuncSetAttribute(const void *k, cudaFuncAttribute, int bytes) {
  if (bytes > 227 * 1024) return cudaErrorInvalidValue;
  limit[{k, device}] = bytes;
  return cudaSuccess;
}
inline cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
inline cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *v, const void *, int, size_t bytes) {
  *v = (int)(228 * 1024 / (bytes + 1024));
  return cudaSuccess;
}
"""

MAIN = r"""
#include <cstddef>
#include "tp_launch.h"
static char ka, kb;
#define CHECK(x) if (!(x)) return __LINE__
int main() {
  int n = 0;
  CHECK(kernel_residency(&ka, 128, 60000, &n) == cudaSuccess && n == 152 * 3);
  CHECK(kernel_residency(&ka, 128, 30000, &n) == cudaSuccess && n == 152 * 7);  // a smaller scene: its own residency,
  CHECK((limit[{&ka, 0}] == 60000));                                            // the limit stays
  CHECK(kernel_residency(&kb, 128, 40000, &n) == cudaSuccess);
  CHECK((limit[{&kb, 0}] == 40000 && limit[{&ka, 0}] == 60000));                // kernels apart
  CHECK(kernel_residency(&ka, 128, 300000, &n) != cudaSuccess);                 // too large: refused,
  CHECK(kernel_residency(&ka, 128, 20000, &n) == cudaSuccess);                  // and the next call works
  CHECK((limit[{&ka, 0}] == 60000));
  device = 1;
  CHECK(kernel_residency(&ka, 128, 20000, &n) == cudaSuccess);
  CHECK((limit[{&ka, 1}] == 20000 && limit[{&ka, 0}] == 60000));                // devices apart
  limit.clear();                                                                // the device was reset
  CHECK(kernel_residency(&ka, 128, 20000, &n) == cudaSuccess);
  CHECK((limit[{&ka, 1}] >= 20000));
  return 0;
}
"""


def test_a_smaller_scene_does_not_lower_the_limit(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "main")
    subprocess.run([gxx, "-std=c++17", "-I", str(tmp_path), "-I", os.path.join(REPO, "imagej-elphel_gb300", "csrc"),
                    str(tmp_path / "main.cpp"), "-o", exe, "-pthread"], check=True)
    assert subprocess.run([exe]).returncode == 0, "failing line of the program"
