"""When a dynamic build empties its creator tables first (csrc/table_state.h).
Builds, replacements and captures in every order of four against the tables
themselves: no build with tables may run on tables that are not empty."""
import os
import subprocess

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include "table_state.h"
// what happens between builds: the arrays replaced (filled with anything), a
// build without tables, one with tables, one that stops midway, a capture of
// a build with tables, a replay of the last capture (refused once the arrays
// were replaced since)
enum { kReplaced, kShallow, kDeep, kStopped, kCapture, kReplay, kOps };
int main() {
  int bad = 0;
  for (int seq = 0; seq < kOps * kOps * kOps * kOps; ++seq) {
    qbc::TableState s;
    bool truly = false;                       // the tables on the device are empty
    bool graph = false, graph_resets = false;
    auto deep = [&](bool stops) {
      const bool reset = s.begin(true);
      if (!truly && !reset) ++bad;
      truly = !stops;
      if (!stops) s.end(true, reset, false);
    };
    for (int k = 0, q = seq; k < 4; ++k, q /= kOps) {
      switch (q % kOps) {
        case kReplaced: s.replaced(); truly = false; graph = false; break;
        case kShallow: { const bool r = s.begin(false); if (r) ++bad; s.end(false, r, false); break; }
        case kDeep: deep(false); break;
        case kStopped: deep(true); break;
        case kCapture: graph_resets = s.begin(true); s.end(true, graph_resets, true); graph = true; break;
        case kReplay:
          if (!graph) break;
          if (!graph_resets && !truly) break;  // a build stopped midway since: a launch failed, and so will this one
          truly = true;
          break;
      }
    }
    deep(false);
  }
  std::printf("%d", bad);
}
"""


def test_no_build_on_tables_left_full(tmp_path):
    src, exe = tmp_path / "tables.cpp", tmp_path / "tables"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "qubatron_gb300", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout == "0"
