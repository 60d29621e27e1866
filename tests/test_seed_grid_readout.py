"""n2w_bvh_seed_grid only copies: the BVH may live on another device than the caller's
current one, on a full device, or beside a stream capture, so reading its grid out neither
launches a kernel nor allocates.  A program stands in for the CUDA runtime's copy, with
host memory for the device's, and records every other call."""
import os
import subprocess

from conftest import PKG, ROOT

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include <vector>
#include "internal.hpp"
#include "n2w.h"

static int g_launches, g_allocations, g_copies;
extern "C" {
cudaError_t cudaMemcpy(void* dst, const void* src, size_t bytes, cudaMemcpyKind) {
  ++g_copies;
  std::memcpy(dst, src, bytes);
  return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t bytes) {
  ++g_allocations;
  *p = nullptr;
  return cudaErrorMemoryAllocation;
}
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) {
  ++g_launches;
  return cudaErrorInvalidDevice;
}
}

int main() {
  n2w_bvh b;
  b.seed_n = 60;
  b.seed_h = 0.25f;
  const int total = 61 * 61 * 61;
  std::vector<int4> cells(total);
  for (int i = 0; i < total; ++i) cells[i] = int4{7 * i + 3, -1, -2, -3};
  b.d_seed = cells.data();
  std::vector<int> slots(total + 1, -9);
  const int rc = n2w_bvh_seed_grid(&b, nullptr, nullptr, nullptr, slots.data());
  bool same = slots[total] == -9;
  for (int i = 0; i < total; ++i) same = same && slots[i] == 7 * i + 3;
  std::printf("rc %d same %d launches %d allocations %d copies %d\n", rc, same, g_launches, g_allocations, g_copies > 0);
  return 0;
}
"""


def test_seed_grid_readout_only_copies(tmp_path):
    src, exe = tmp_path / "readout.cpp", tmp_path / "readout"
    src.write_text(PROGRAM)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O1", "-rdynamic", f"-I{ROOT / 'include'}", f"-I{PKG / 'csrc'}", f"-I{cuda}/include",
                    str(src), "-o", str(exe), f"-L{PKG / 'lib'}", "-ln2w", f"-Wl,-rpath,{PKG / 'lib'}",
                    f"-L{cuda}/lib64", "-lcudart"], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    assert out.strip() == "rc 0 same 1 launches 0 allocations 0 copies 1", out
