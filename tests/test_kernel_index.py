"""The numbers by which a context remembers the kernels whose attributes it
has set (csrc/kernel_index.h): one per kernel, all below their count."""
import os
import subprocess

from conftest import ROOT

PROGRAM = r"""
#include <bitset>
#include <cstdio>
#include "kernel_index.h"
int main() {
  std::bitset<qbc::kKernels> seen;
  auto take = [&](int i) {
    if (i < 0 || i >= qbc::kKernels || seen[i]) std::printf("index %d: %s\n", i, i < 0 || i >= qbc::kKernels ? "outside" : "taken");
    else seen[i] = true;
  };
  for (int k = 0; k < 4; ++k) {
    for (int walk = 0; walk < qbc::kWalkKinds; ++walk) {
      for (int mode = 0; mode < qbc::kModeKinds; ++mode) take(qbc::render_kernel_index(k & 1, k & 2, mode, false, walk));
      take(qbc::render_kernel_index(k & 1, k & 2, 2, true, walk));  // the shade pass with proposals
    }
    take(qbc::simple_kernel_index(k & 1, k & 2));
  }
  if (!seen.all()) std::printf("%d numbers unused\n", (int)(qbc::kKernels - seen.count()));
}
"""


def test_one_number_per_kernel(tmp_path):
    src, exe = tmp_path / "index.cpp", tmp_path / "index"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "qubatron_gb300", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout == ""
