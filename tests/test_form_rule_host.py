"""The memory rule of the default sweep form, for a handle before and after its buffers
exist: the same answer."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "form_rule.h"
using ouranos::edges_crowd;
int main() {
  const size_t mb = 1 << 20, fluxes = 1640 * mb, nominal = 26 * mb, edges = 102 * mb;
  for (size_t device = 2000 * mb; device < 9000 * mb; device += 100 * mb) {
    const bool fresh = edges_crowd(edges, nominal, fluxes, device, 0);
    if (fresh != (edges + fluxes > device / 2)) return 1;
    // the schedule's edges, then the fluxes of the first sweep
    if (device > edges && edges_crowd(edges, nominal, fluxes, device - edges, edges) != fresh) return 2;
    if (device > edges + fluxes && edges_crowd(edges, nominal, fluxes, device - edges - fluxes, edges + fluxes) != fresh)
      return 3;
    if (edges_crowd(nominal, nominal, fluxes, 0, 0)) return 4;  // (no smaller tiles)
  }
}
"""


def test_the_rule_does_not_count_the_handles_own_buffers_twice(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    src = tmp_path / "form_rule.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "form_rule")
    subprocess.run([cxx, "-std=c++17", "-I", os.path.join(ROOT, "ouranos_gb300", "csrc"), str(src), "-o", exe],
                   check=True)
    assert subprocess.run([exe]).returncode == 0
