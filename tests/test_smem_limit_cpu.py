"""The dynamic shared-memory limit of a kernel (set_smem) is one value per
function and device, and separate fleets, shards and the server launch from
separate host threads: a call for a small launch must not lower the limit
another thread has just raised for a larger one.  The header is compiled with
the two runtime calls it makes replaced by fakes that hold the limits."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

SOURCE = r"""
#include <cuda_runtime.h>
#include <atomic>
#include <cstdio>
#include <thread>
static thread_local int t_dev = 0;
static std::atomic<size_t> g_limit[2][2];  // [device][kernel]
__global__ void k0() {}
__global__ void k1() {}
static cudaError_t fake_get_device(int* d) { *d = t_dev; return cudaSuccess; }
static cudaError_t fake_set(const void* f, cudaFuncAttribute, int v) {
  if (v > 227 * 1024) return cudaErrorInvalidValue;
  g_limit[t_dev][f == (const void*)k1] = (size_t)v;
  return cudaSuccess;
}
#define cudaGetDevice fake_get_device
#define cudaFuncSetAttribute fake_set
#include "kernels.cuh"
using dnspir::set_smem;
#define CHECK(c) do { if (!(c)) { printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
int main() {
  set_smem(k0, 118784);
  set_smem(k0, 82960);  // a smaller launch of the same kernel
  CHECK(g_limit[0][0] == 118784);
  set_smem(k1, 82960);
  CHECK(g_limit[0][1] == 82960);
  t_dev = 1;            // the limit belongs to the device's copy of the function
  set_smem(k0, 82960);
  CHECK(g_limit[1][0] == 82960);
  set_smem(k0, 300000);  // refused: the launch reports it, and a later fitting size still goes through
  set_smem(k0, 200000);
  CHECK(g_limit[1][0] == 200000);
  std::atomic<int> bad(0);
  auto user = [&](size_t bytes) {
    t_dev = 0;
    for (int i = 0; i < 200000; i++) {
      set_smem(k1, bytes);
      if (g_limit[0][1] < bytes) bad++;  // the launch that follows would be refused
    }
  };
  std::thread a(user, 55296), b(user, 73728), c(user, 118784);
  a.join(), b.join(), c.join();
  CHECK(bad == 0);
  return 0;
}
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="needs nvcc")
def test_limit_is_never_lowered(tmp_path):
    src, exe = tmp_path / "limit.cu", tmp_path / "limit"
    src.write_text(SOURCE)
    subprocess.check_call([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                           "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "dnspir_b200", "csrc"),
                           "-o", str(exe), str(src)])
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
