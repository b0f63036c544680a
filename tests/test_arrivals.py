"""The counting of the resident optimiser's grid barrier (csrc/arrivals.h) on the CPU: no block may pass a round before all
have arrived, and all must once they have, also in the rounds in which the 32-bit count wraps."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <initializer_list>
#include "arrivals.h"
using namespace pacmap;
int main() {
  for (uint32_t blocks : {1u, 2u, 63u, 148u, 444u, 592u}) {
    const uint64_t wraps = 4294967296ull / blocks;
    for (uint64_t base : {uint64_t(1), wraps - 4, 2 * wraps - 4, 5 * wraps - 4})
      for (uint64_t round = base; round < base + 12; ++round) {
        // true count of arrivals, in 64 bits; the kernel's counter is its low word from ARRIVALS_START on
        const uint32_t want = arrivals_wanted(static_cast<uint32_t>(round), blocks);
        for (uint64_t missing = 1; missing <= blocks; ++missing)
          if (arrivals_reached(static_cast<uint32_t>(ARRIVALS_START + round * blocks - missing), want))
            return std::printf("passes early: %u blocks, round %llu\n", blocks, (unsigned long long)round), 1;
        for (uint64_t ahead = 0; ahead < blocks; ++ahead)  // others may already be in the next round
          if (!arrivals_reached(static_cast<uint32_t>(ARRIVALS_START + round * blocks + ahead), want))
            return std::printf("waits on: %u blocks, round %llu\n", blocks, (unsigned long long)round), 1;
      }
  }
  return 0;
}
"""


def test_no_block_passes_early_where_the_count_wraps(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    cxx = os.environ.get("PACMAP_HOST_CXX", "/usr/bin/g++")
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "pacmap-rs_b200", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
