"""The once-per-device kernel attributes of the launchers, on the host with a stand-in for the CUDA call."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "csrc"
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

PROGRAM = r"""
#include <cuda_runtime.h>
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>
static std::atomic<int> g_set{0}, g_fail{0};
template <typename K> cudaError_t slow_set(K*, cudaFuncAttribute, int) {
  std::this_thread::sleep_for(std::chrono::milliseconds(100));
  if (g_fail.load()) return cudaErrorInvalidValue;
  ++g_set;
  return cudaSuccess;
}
#define cudaFuncSetAttribute slow_set
#include "pnm_internal.h"
static thread_local int t_dev = 0;
int pnm::current_device() { return t_dev; }
static void kernel(int) {}
int main() {
  pnm::DeviceMask mask{0};
  g_fail = 1;
  if (pnm::allow_smem(kernel, 1, mask)) return 1;          // a call that failed is made again
  g_fail = 0;
  std::atomic<int> early{0};
  std::vector<std::thread> all;
  for (int i = 0; i < 8; ++i)
    all.emplace_back([&, i] {
      std::this_thread::sleep_for(std::chrono::milliseconds(10 * i));
      if (!pnm::allow_smem(kernel, 1, mask) || g_set.load() == 0) ++early;      // may launch before the attribute is set
    });
  for (auto& t : all) t.join();
  const int before = g_set.load();
  if (!pnm::allow_smem(kernel, 1, mask) || g_set.load() != before) return 2;    // once per device ...
  t_dev = 1;
  if (!pnm::allow_smem(kernel, 1, mask) || g_set.load() != before + 1) return 3;   // ... and on every device
  return early.load() ? 4 : 0;
}
"""


@pytest.mark.skipif(not Path(NVCC).exists(), reason="no nvcc")
def test_no_thread_launches_before_the_attribute_is_set(tmp_path):
    src = tmp_path / "first_use.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "first_use"
    built = subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(CSRC), "-Xcompiler", "-pthread",
                            "-o", str(exe), str(src)], capture_output=True, text=True)
    assert built.returncode == 0, built.stderr[-2000:]
    assert subprocess.run([str(exe)], timeout=60).returncode == 0
