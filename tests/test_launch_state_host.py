"""The sweep kernels' launch settings against a fake runtime with two devices: the
runtime keeps a function's attributes per device, so each device gets its own."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <map>
#include <utility>
#include "launch_state.h"
static int current = 0, opt_ins = 0;
static const int kSms[2] = {152, 76};
static std::map<std::pair<int, int>, int> attr;  // (device, attribute) -> value
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int d) {
  *v = a == cudaDevAttrMultiProcessorCount ? kSms[d] : 228 * 1024;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute a, int v) {
  attr[{current, (int)a}] = v;
  opt_ins += a == cudaFuncAttributeMaxDynamicSharedMemorySize;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) {
  *n = 3;
  return cudaSuccess;
}
}
static bool launch(ouranos::SweepLaunch& st, int dev, int arrays, int grid) {
  current = dev;
  const size_t smem = 40000 * arrays;
  if (st.prepare(nullptr, arrays, grid, 128, smem, 80000, 0, 64) != cudaSuccess) return false;
  // what the runtime would check at the launch, and the carveout of this device's grid
  const int per_sm = (grid + kSms[dev] - 1) / kSms[dev] < 3 ? (grid + kSms[dev] - 1) / kSms[dev] : 3;
  const long room = (228 - 64) * 1024, fit = room / (long)(smem + 1024);
  const long need = (per_sm < fit ? per_sm : fit) * (long)(smem + 1024);
  return attr[{dev, (int)cudaFuncAttributeMaxDynamicSharedMemorySize}] >= (int)smem &&
         attr[{dev, (int)cudaFuncAttributePreferredSharedMemoryCarveout}] == (int)((need * 100 + 228 * 1024 - 1) / (228 * 1024));
}
int main() {
  static ouranos::SweepLaunch st;
  for (int round = 0; round < 2; ++round)
    for (int dev : {0, 1, 0})
      for (int arrays : {2, 1})
        if (!launch(st, dev, arrays, 152)) return std::printf("device %d arrays %d\n", dev, arrays), 1;
  return opt_ins == 4 ? 0 : 2;  // (once per device and number of arrays)
}
"""


def test_settings_are_kept_per_device(tmp_path):
    cxx = shutil.which("g++")
    cuda = "/usr/local/cuda/include"
    if not cxx or not os.path.exists(os.path.join(cuda, "cuda_runtime_api.h")):
        pytest.skip("no host compiler or CUDA headers")
    src = tmp_path / "launch_state.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "launch_state")
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "ouranos_gb300", "csrc"), "-isystem", cuda,
                    str(src), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
