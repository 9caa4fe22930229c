"""The cache of resident block counts (csrc/resident.h): one entry per kernel, device, block size
and shared memory.  The marching slow tendency asks for 128 to 256 threads of one kernel,
depending on the grid, and splits its work by the count."""
import subprocess
from pathlib import Path

from oraclev8_b200 import build as B

SOURCE = r"""
#include <cstdio>
#include "resident.h"
int main() {
  ob::ResidentCache c;
  int asked = 0, wrong = 0;
  const char k[2] = {};
  for (int pass = 0; pass < 2; ++pass)
    for (int kernel = 0; kernel < 2; ++kernel)
      for (int dev = 0; dev < 2; ++dev)
        for (int threads : {128, 160, 256})
          for (std::size_t smem : {std::size_t(0), std::size_t(1024)}) {
            const int want = 1000 * kernel + 100 * dev + 2048 / threads + (smem ? 20 : 0);
            wrong += want != c.get(k + kernel, dev, threads, smem, [&] { ++asked; return want; });
          }
  std::printf("%d %d\n", wrong, asked);
  return 0;
}
"""


def test_counts_are_kept_by_block_size_and_shared_memory(tmp_path: Path):
    src, exe = tmp_path / "resident.cpp", tmp_path / "resident"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-I", str(B.CSRC), "-o", str(exe), str(src)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out == "0 24\n"
