"""Build the in-tree CUDA library ``liboracle_b200.so`` for sm_100a.

    python -m oraclev8_b200.build            # or: python oraclev8_b200/build.py

The library has a plain C ABI (include/oracle_b200.h) and no dependency on
PyTorch; the Python layer loads it with ctypes.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import tempfile
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
ROOT = PKG.parent
CSRC = PKG / "csrc"
LIB = PKG / "liboracle_b200.so"
# translation units: (source, defines), compiled side by side
UNITS = [(CSRC / "api.cu", ())] + [
    (CSRC / "zfft.cu", (f"-DOB_ZREAL={real}", f"-DOB_ZELEM={elem}", f"-DOB_ZPART={part}"))
    for real, elem in (("float", 4), ("double", 8)) for part in (0, 2, 4, 6, 8)]
DEPS = (sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh")) + sorted(CSRC.glob("*.h"))
        + [ROOT / "include" / "oracle_b200.h"])

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
FLAGS = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "-Xptxas", "-warn-spills"]


def nvcc() -> str:
    for c in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if c and Path(c).exists():
            return c
    raise RuntimeError("nvcc not found; the CUDA toolkit is required to build oraclev8_b200")


def up_to_date() -> bool:
    if not LIB.exists():
        return False
    t = LIB.stat().st_mtime
    return all(d.stat().st_mtime <= t for d in DEPS)


def build(force: bool = False, verbose: bool = False) -> Path:
    if not force and up_to_date():
        return LIB
    tmp = LIB.with_suffix(".so.tmp")
    flags = FLAGS + (["-Xptxas=-v"] if verbose else [])
    with tempfile.TemporaryDirectory() as d:
        def unit(i):
            src, defines = UNITS[i]
            obj = Path(d) / f"{src.stem}_{i}.o"
            cmd = [nvcc(), *ARCH, *flags, *defines, "-c", "-o", str(obj), str(src)]
            if verbose:
                print(" ".join(cmd), flush=True)
            subprocess.run(cmd, check=True)
            return str(obj)

        with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as pool:
            objs = list(pool.map(unit, range(len(UNITS))))
        subprocess.run([nvcc(), *ARCH, "-shared", "-o", str(tmp), *objs, "-lcudart"], check=True)
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(LIB)
