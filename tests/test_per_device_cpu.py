"""One-time kernel setup is made on every device that a process uses: the helper against a stand-in for the CUDA runtime,
and no kernel attribute set behind a process-wide flag."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "tnpy_gb300" / "csrc"

RUNTIME = """
#pragma once
#include <cstddef>
enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1 };
enum cudaFuncAttribute { cudaFuncAttributeMaxDynamicSharedMemorySize = 8 };
extern thread_local int current_device;
extern int calls[128], last[128];
extern bool refuse;
inline cudaError_t cudaGetDevice(int* d) { *d = current_device; return cudaSuccess; }
template <typename K>
cudaError_t cudaFuncSetAttribute(K, cudaFuncAttribute, int value) {
  if (refuse) return cudaErrorInvalidValue;
  ++calls[current_device];
  last[current_device] = value;
  return cudaSuccess;
}
"""

PROGRAM = """
#include "per_device.cuh"
#include <cassert>
#include <thread>
#include <vector>
thread_local int current_device = 0;
int calls[128], last[128];
bool refuse = false;
void kernel(int) {}
tnx::DeviceSet allowed, other;
int main() {
  for (int dev : {0, 1, 0, 3, 1, 63}) {
    current_device = dev;
    assert(tnx::allow_smem(kernel, 70000, allowed) == cudaSuccess);
  }
  for (int dev : {0, 1, 3, 63}) assert(calls[dev] == 1 && last[dev] == 70000);
  assert(calls[2] == 0);
  current_device = 2;  // a failed setup is not remembered
  refuse = true;
  assert(tnx::allow_smem(kernel, 70000, allowed) == cudaErrorInvalidValue);
  refuse = false;
  assert(tnx::allow_smem(kernel, 70000, allowed) == cudaSuccess && calls[2] == 1);
  current_device = 100;  // beyond the set: each time
  for (int i = 0; i < 3; ++i) assert(tnx::allow_smem(kernel, 70000, allowed) == cudaSuccess);
  assert(calls[100] == 3);
  current_device = 0;  // another kernel's set
  assert(tnx::allow_smem(kernel, 80000, other) == cudaSuccess && calls[0] == 2 && last[0] == 80000);
  tnx::DeviceSet shared;
  std::vector<std::thread> threads;
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([&shared, t] {
      current_device = 10 + t;
      for (int i = 0; i < 100; ++i) assert(tnx::allow_smem(kernel, 50000, shared) == cudaSuccess);
    });
  for (auto& t : threads) t.join();
  for (int t = 0; t < 8; ++t) assert(calls[10 + t] == 1 && shared.has(10 + t));
  return 0;
}
"""


def test_setup_is_made_once_on_each_device(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "main.cpp").write_text(PROGRAM)
    exe = tmp_path / "main"
    subprocess.run([gxx, "-std=c++17", "-pthread", "-I", str(tmp_path), "-I", str(CSRC), str(tmp_path / "main.cpp"), "-o",
                    str(exe)], check=True)
    subprocess.run([str(exe)], check=True, timeout=60)


@pytest.mark.parametrize("path", sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]), ids=lambda p: p.name)
def test_no_kernel_attribute_behind_a_process_wide_flag(path):
    text = path.read_text()
    for m in re.finditer(r"cudaFuncSetAttribute\(", text):
        before = text[: m.start()][-900:]
        assert "atomic<bool>" not in before
        if "call_once" in before:
            assert re.search(r"call_once\(once\[dev\]", before)
