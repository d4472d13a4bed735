"""The epilogue walk of the tensor-core GEMM's split tiles (csrc/tc_pieces.h), compiled for the host:
whatever clusters give up waiting, and from whichever item on, every counter is zero when the launch
has ended, as the next launch expects it; and where none gives up, every whole tile is stored once
and every split tile summed once, after all of its pieces have been stored."""

import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "finitemptools_gb300", "csrc")

PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
#include "tc_pieces.h"
using namespace fmpt::tc;

int main() {
  std::mt19937 rng(7);
  auto pick = [&](int lo, int hi) { return lo + (int)(rng() % (unsigned)(hi - lo + 1)); };
  for (int trial = 0; trial < 20000; trial++) {
    const int S = pick(2, 4), ncl0 = pick(1, 76), tail = pick(1, std::max(1, ncl0 / S));
    PairSched sp{ncl0 * pick(0, 3), tail, S, nullptr, nullptr};
    const int items = sp.full + tail * S, ncl = std::min(items, ncl0), nk = pick(4 * S, 60);
    const bool faults = trial % 2;
    std::vector<int> count(tail, 0), stored(sp.full, 0), pieces(tail, 0), sums(tail, 0);
    std::vector<int> counted(tail, 0), order(ncl);
    for (int i = 0; i < ncl; i++) order[i] = i;
    std::shuffle(order.begin(), order.end(), rng);
    for (int cl : order) {
      const int stop = faults && rng() % 3 == 0 ? pick(0, 3) : 1 << 30;
      pair_epilogue(
          sp, cl, ncl, nk, [&](int local) { return local < stop; },
          [&](int local, int u, int t) {
            if (local >= stop) std::exit(1);
            if (t < 0) stored[u]++; else pieces[u - sp.full]++;
          },
          [&](int ut) { counted[ut]++; return count[ut]++ == S - 1; },
          [&](int ut, int u) {
            if (u != sp.full + ut || (!faults && pieces[ut] != S)) std::exit(2);
            sums[ut]++;
          },
          [&](int ut) { count[ut] = 0; });
    }
    for (int i = 0; i < tail; i++) {
      if (count[i] != 0 || counted[i] != S) return 3;
      if (!faults && sums[i] != 1) return 4;
    }
    if (!faults)
      for (int n : stored) if (n != 1) return 5;
  }
  std::puts("ok");
  return 0;
}
"""


def test_counters_return_to_zero(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("needs a host C++ compiler")
    src, exe = tmp_path / "walk.cpp", tmp_path / "walk"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0 and run.stdout == "ok\n", run.returncode
