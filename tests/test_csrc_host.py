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


def test_kernel_setup_is_per_device(tmp_path):
    """A second device, kernel or size is set up for itself, each once however
    many threads ask; a set-up that failed is tried again."""
    out = _run(tmp_path, r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.h"
int main() {
  static pcc::PerDevice cache;
  static int kernels[2];
  std::atomic<int> made{0}, wrong{0};
  int v = 7;
  wrong += cache.Get(0, &kernels[0], 64, &v, [&](int*) { return false; });
  std::vector<std::thread> all;
  for (int t = 0; t < 16; ++t)
    all.emplace_back([&] {
      for (int device = 0; device < 3; ++device)
        for (int k = 0; k < 2; ++k)
          for (int size : std::vector<int>{64, 96}) {
            int got = 0;
            wrong += !cache.Get(device, &kernels[k], size, &got, [&](int* n) {
              ++made;
              *n = device * 1000 + k * 100 + size;
              return true;
            });
            wrong += got != device * 1000 + k * 100 + size;
          }
    });
  for (auto& t : all) t.join();
  std::printf("%d %d\n", made.load(), wrong.load());
}
""")
    assert out.split() == ["12", "0"]
