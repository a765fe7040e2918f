"""The fixed-point sum of 32 FP32 values (a warp's share of the diffusion CG's sums)
against exactly rounded sums: at least the accuracy of sums in FP64."""
import math
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "fsum.cuh"
int main() {
  unsigned b[32];
  while (std::fread(b, 4, 32, stdin) == 32) {
    unsigned top = 0;
    for (unsigned v : b) top = top > (v & 0x7fffffffu) ? top : v & 0x7fffffffu;
    const int e = ouranos::fixed_exponent(top);
    long long s = 0;
    for (unsigned v : b) s += ouranos::fixed_of(v, e);
    std::printf("%a\n", ouranos::fixed_value(s, e));
  }
}
"""


def _groups():
    rng = np.random.default_rng(1)
    n = 400
    f = np.float32
    yield rng.standard_normal((n, 32)).astype(f)
    yield (rng.standard_normal((n, 32)) * 2.0 ** rng.uniform(-60, 60, (n, 32))).astype(f)
    x = rng.standard_normal((n, 32)).astype(f)
    x[:, 16:] = -x[:, :16] * (1 + f(2e-7) * rng.integers(0, 2, (n, 16)).astype(f))  # all but cancels
    yield x
    yield (rng.integers(-3, 4, (n, 32)) * 2.0 ** -149).astype(f)                    # denormals, zeros
    yield (rng.uniform(-1, 1, (n, 32)) * 2.0 ** -125).astype(f)                     # around the smallest normal
    yield np.where(rng.integers(0, 2, (n, 32)), f(3.4028235e38), f(-1.5e38)).astype(f)
    yield np.full((4, 32), f(3.4028235e38))
    yield np.full((4, 32), f(-3.4028235e38))
    yield np.zeros((2, 32), f)


def test_sum_of_a_warp(tmp_path):
    cxx = shutil.which("g++")
    cuda = "/usr/local/cuda/include"
    if not cxx or not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("no host compiler or CUDA headers")
    src = tmp_path / "fsum.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "fsum")
    subprocess.run([cxx, "-std=c++17", "-O2", "-I", os.path.join(ROOT, "ouranos_gb300", "csrc"), "-isystem", cuda,
                    str(src), "-o", exe], check=True)
    x = np.concatenate(list(_groups()))
    out = subprocess.run([exe], input=x.tobytes(), capture_output=True, check=True).stdout.split()
    assert len(out) == len(x)
    for row, got in zip(x.astype(np.float64), out):
        got = float.fromhex(got.decode())
        exact = math.fsum(row)
        # one rounding to FP64, and at most 2^-57 of the largest value cut off from each
        assert abs(got - exact) <= 2.0 ** -53 * abs(exact) + 32 * 2.0 ** -57 * np.abs(row).max()
