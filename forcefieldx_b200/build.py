"""Build libffxcuda.so (the energy library) and libffxpeak.so (FMA-throughput microkernels
for the benchmark's pipe fractions) in-tree with nvcc for sm_100a (no JIT cache, no torch
extension)."""
from __future__ import annotations

import os
import subprocess
import sys
import tempfile
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
SOURCES = ["handle.cu", "nlist.cu", "pme.cu", "real.cu", "vdw.cu", "recip.cu", "pcg.cu", "md.cu", "batch.cu"]
LIB = os.path.join(HERE, "libffxcuda.so")
PEAK_SRC = "peak.cu"
PEAK_LIB = os.path.join(HERE, "libffxpeak.so")
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
              "-diag-suppress", "177"]
# Sources without line tables.  Those of the unrolled transforms are 13 of their module's 17 MB,
# which a process's first handle would load: creating it and its first evaluation took 40 ms
# instead of 25 (648 atoms FP64).
NO_LINE_TABLES = {"pme.cu"}


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def compile_flags(source: str) -> list:
    return NVCC_FLAGS + ([] if source in NO_LINE_TABLES else ["-lineinfo"])


def stale() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(HERE, "csrc", s) for s in SOURCES + ["ffx_internal.cuh", "launch.cuh", "fft.cuh"]]
    deps += [os.path.abspath(__file__), os.path.join(os.path.dirname(HERE), "include", "ffxcuda.h")]
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    def run(cmd):
        if verbose:
            print(" ".join(cmd), file=sys.stderr)
        subprocess.run(cmd, check=True)

    peak_src = os.path.join(HERE, "csrc", PEAK_SRC)
    if force or not os.path.exists(PEAK_LIB) or os.path.getmtime(PEAK_LIB) < os.path.getmtime(peak_src):
        run([nvcc()] + compile_flags(PEAK_SRC) + ["-shared", "-o", PEAK_LIB, peak_src])
    if not force and not stale():
        return LIB
    with tempfile.TemporaryDirectory() as tmp, ThreadPoolExecutor(8) as pool:
        objects = [os.path.join(tmp, s + ".o") for s in SOURCES]
        list(pool.map(lambda s, o: run([nvcc()] + compile_flags(s) + ["-c", "-o", o, os.path.join(HERE, "csrc", s)]),
                      SOURCES, objects))
        run([nvcc()] + NVCC_FLAGS + ["-shared", "-o", LIB] + objects)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
