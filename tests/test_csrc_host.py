"""CPU tests of the library's host arithmetic: headers of csrc/ that a host
compiler takes, each driven by a small program."""

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "parallel-correlation-clustering_gb300", "csrc")


def _run(tmp_path, source):
    src, exe = tmp_path / "t.cc", tmp_path / "t"
    src.write_text(source)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-pthread", "-I" + CSRC, "-o", str(exe), str(src)],
                   check=True)
    return subprocess.run([str(exe)], check=True, stdout=subprocess.PIPE, text=True).stdout


def test_barrier_count_passes_2_32(tmp_path):
    """Every barrier of a long run: not reached while a CTA is missing, reached
    with the last one and while the others go on to the next, on both sides
    of 2^32."""
    out = _run(tmp_path, r"""
#include <cstdio>
#include <initializer_list>
#include "barrier.h"
int main() {
  int bad = 0;
  for (uint32_t grid : {2u, 37u, 304u, 1024u}) {
    for (uint32_t start : {pcc::kBarrierStart, 0u, 0u - 3u * grid, 0x80000000u - 2u * grid}) {
      uint32_t target = start;
      for (int round = 0; round < 4000; ++round) {
        const uint32_t before = target;
        target += grid;
        for (uint32_t here = 0; here < grid; ++here) bad += pcc::BarrierReached(before + here, target);
        for (uint32_t ahead = 0; ahead < grid; ++ahead) bad += !pcc::BarrierReached(target + ahead, target);
      }
    }
  }
  std::printf("%d\n", bad);
}
""")
    assert out.strip() == "0"
