"""The rule that lets a call's level pairs move as one access each (csrc/zfft.h, zpairs),
compiled for the host: an even level count and every field on a multiple of the pair."""
import subprocess
from pathlib import Path

from oraclev8_b200 import build as B

SOURCE = r"""
#include <cstdio>
#include "zfft.h"
using ob::zpairs;
template <class T>
int bad() {
  alignas(64) static unsigned char buf[256];
  auto at = [](int n) { return reinterpret_cast<const T*>(buf) + n; };  // n elements in
  const T* none = nullptr;
  int n = 0;
  for (int i = 0; i < 8; ++i)
    for (int j = 0; j < 8; ++j)
      for (int nz = 3; nz < 9; ++nz)
        n += zpairs<T>(nz, at(i), at(j), none) != (nz % 2 == 0 && i % 2 == 0 && j % 2 == 0);
  return n;
}
int main() {
  std::printf("%d %d\n", bad<float>(), bad<double>());
  return 0;
}
"""


def test_pairs_only_of_even_columns_on_pair_boundaries(tmp_path: Path):
    src, exe = tmp_path / "pairs.cu", tmp_path / "pairs"
    src.write_text(SOURCE)
    subprocess.run([B.nvcc(), *B.ARCH, "-std=c++17", "-I", str(B.CSRC), "-o", str(exe), str(src)],
                   check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout == "0 0\n"
