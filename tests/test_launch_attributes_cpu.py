"""Host side of the launchers: the once-per-device kernel attributes (with a stand-in for the CUDA call) and the LayerNorm plan."""
import re
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


PLAN = r"""
#include <cstdio>
#include "norm.cuh"
using namespace pnm;
int main() {
  const int sms = 148;
  for (int C = 8; C <= 1024; C += 8)
    for (long long M : {1LL, 7LL, 100LL, 3551LL, 10656LL, 14207LL, 14208LL, 60001LL, 113663LL, 113664LL, 1000000LL, 3000000LL})
      for (int tensors = 1; tensors <= 3; ++tensors)
        for (int backward = 0; backward < 2; ++backward) {
          if (tensors == (backward ? 1 : 3)) continue;
          const int least = backward ? ln_bwd_rows(C) : kLnWarps * (C <= 256 ? 2 : 1);
          const int per_sm = backward ? ln_bwd_per_sm(C) : (C <= 512 ? 3 : 2);
          const LnStream p = ln_stream_plan(M, C, tensors, least, per_sm, sms);
          const long long ring = 1LL * p.stages * p.rows * C * 2 * tensors;
          const bool ok = p.rows >= least && p.rows % least == 0 && p.stages >= 2 && p.stages <= 8 && p.grid >= 1 &&
                          p.smem >= ring + 16 * p.stages + 8 && (!backward || p.smem >= kLnFoldBytes + 16 * p.stages + 8) &&
                          p.smem <= kLnSmemMax && 1LL * per_sm * (p.smem + 1024) <= 228 * 1024 &&   // all CTAs of the grid are resident
                          p.grid <= sms * per_sm && (!backward || p.grid <= layernorm_bwd_grid(M, sms, C));
          if (!ok) return printf("C %d M %lld tensors %d backward %d: rows %d stages %d grid %d smem %d\\n", C, M, tensors, backward, p.rows,
                                 p.stages, p.grid, p.smem), 1;
        }
  return 0;
}
"""


def _run(tmp_path, program):
    src, exe = tmp_path / "program.cu", tmp_path / "program"
    src.write_text(program)
    built = subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(CSRC), "-Xcompiler", "-pthread",
                            "-o", str(exe), str(src)], capture_output=True, text=True)
    assert built.returncode == 0, built.stderr[-2000:]
    done = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert done.returncode == 0, done.stdout


@pytest.mark.skipif(not Path(NVCC).exists(), reason="no nvcc")
def test_no_thread_launches_before_the_attribute_is_set(tmp_path):
    _run(tmp_path, PROGRAM)


@pytest.mark.skipif(not Path(NVCC).exists(), reason="no nvcc")
def test_layernorm_plans_fit_the_sm(tmp_path):
    _run(tmp_path, PLAN)


@pytest.mark.skipif(not Path(NVCC).exists(), reason="no nvcc")
@pytest.mark.parametrize("budget,compiles", [("2000000000ull", True), ("5000000000ull", False)])
def test_a_wait_budget_that_the_timers_low_word_cannot_hold_does_not_compile(tmp_path, budget, compiles):
    text = (CSRC / "common.cuh").read_text()
    assert "kWaitBudgetNs = 2000000000ull" in text
    (tmp_path / "common.cuh").write_text(text.replace("kWaitBudgetNs = 2000000000ull", f"kWaitBudgetNs = {budget}"))
    (tmp_path / "unit.cu").write_text('#include "common.cuh"\n')
    built = subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(tmp_path), "-I", str(CSRC), "-c",
                            "-o", str(tmp_path / "unit.o"), str(tmp_path / "unit.cu")], capture_output=True, text=True)
    assert (built.returncode == 0) == compiles and (compiles or "low word" in built.stdout + built.stderr)


@pytest.mark.parametrize("name", ["gemm_tn.cuh", "gemm_tn_pair.cuh", "gemm_nt.cuh", "gemm_nt_pair.cuh", "conv3_wgrad.cuh", "afno_rows_tc.cuh"])
def test_whole_warps_take_the_end_of_a_wait_together(name):
    """An epilogue warp goes on to elect.sync and TMEM loads, for which its lanes must be together: also where a wait ran out, which no
    test can bring about."""
    waits = re.findall(r"\b(mbar_wait\w*)\(&?(?:tfull|mybar)\b", (CSRC / name).read_text())
    assert waits and set(waits) == {"mbar_wait_warp"}
