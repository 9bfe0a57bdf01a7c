"""The progress counters of the persistent batch kernel are 32 bits and go round in long launches: the
comparison that a waiting warp makes, compiled for the host, around the wrap."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "ecmc-qncb_b200" / "csrc"

PROGRAM = r"""
#include "counter.h"
#include <cstdio>
// A lattice of `tiles` tiles a level, levels around the one at which its counter of finished tiles passes
// 2^32: a tile of level k may start when all k * tiles earlier ones are finished, not before.
int main() {
  const uint32_t sizes[] = {1u, 4u, 3001u, 16384u, 262144u, 1u << 24};
  for (uint32_t tiles : sizes) {
    const uint32_t wrap = (uint32_t)((1ull << 32) / tiles);
    for (uint32_t level = wrap < 3 ? 1 : wrap - 3; level < wrap + 4u && level != 0; ++level) {
      const uint32_t target = level * tiles;
      const uint64_t finished = (uint64_t)level * tiles;
      if (!qcb::counter_reached((uint32_t)finished, target)) return std::printf("waits for nothing: %u %u\n", tiles, level), 1;
      if (!qcb::counter_reached((uint32_t)(finished + tiles - 1), target)) return std::printf("lost: %u %u\n", tiles, level), 1;
      if (qcb::counter_reached((uint32_t)(finished - 1), target)) return std::printf("starts early: %u %u\n", tiles, level), 1;
      if (qcb::counter_reached((uint32_t)(finished - tiles), target)) return std::printf("a level early: %u %u\n", tiles, level), 1;
    }
  }
  return 0;
}
"""


def test_comparison_around_the_wrap(tmp_path):
    src, exe = tmp_path / "wrap.cpp", tmp_path / "wrap"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
