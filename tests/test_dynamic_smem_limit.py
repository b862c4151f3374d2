"""Two threads that ask for different amounts of a kernel's dynamic shared memory at the same time: the limit ends at the larger one,
and neither returns while it is below what it asked for (the header's own function, compiled for the host with the CUDA calls
replaced)."""
import shutil
import subprocess

import pytest

from d2conv3d_b200 import build

PROGRAM = r"""
#include <cuda_runtime.h>
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>
static std::atomic<int> limit{0};
static std::atomic<bool> small_inside{false};
static void pause_ms(int ms) { std::this_thread::sleep_for(std::chrono::milliseconds(ms)); }
static cudaError_t fake_get_device(int* dev) { *dev = 0; return cudaSuccess; }
template <typename F>
static cudaError_t fake_set(F*, cudaFuncAttribute, int bytes) {
  if (bytes < 60000) {             // the smaller request takes long, so that the larger one overtakes it if it can
    small_inside = true;
    pause_ms(300);
  }
  limit = bytes;
  return cudaSuccess;
}
#define cudaGetDevice fake_get_device
#define cudaFuncSetAttribute fake_set
#include "d2c_common.cuh"
namespace d2c { void set_last_cuda_error(cudaError_t) {} }
__global__ void kernel() {}
int main() {
  int at_small = 0, at_large = 0, bad = 0;
  std::thread a([&] { bad += d2c::allow_dynamic_smem<kernel>(50000); at_small = limit; });
  while (!small_inside) pause_ms(1);
  std::thread b([&] { bad += d2c::allow_dynamic_smem<kernel>(65000); pause_ms(600); at_large = limit; });
  a.join();
  b.join();
  bad += d2c::allow_dynamic_smem<kernel>(40000);
  printf("%d %d %d %d\n", bad, at_small, at_large, (int)limit);
}
"""


def test_limit_never_goes_down(tmp_path):
    nvcc = build._nvcc()
    if shutil.which(nvcc) is None:
        pytest.skip("needs nvcc")
    src, exe = tmp_path / "limit.cu", tmp_path / "limit"
    src.write_text(PROGRAM)
    flags = [f for f in build.NVCC_FLAGS if f != "-O3"]
    subprocess.run([nvcc] + flags + ["-I", build.CSRC, "-o", str(exe), str(src)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout
    bad, at_small, at_large, last = map(int, out.split())
    assert bad == 0
    assert at_small >= 50000 and at_large == last == 65000
