"""Builds of single sources in which every bounded wait gives up when its first poll fails, so that a
test sees what a wait that runs out reports, on a GPU that is in order."""
import ctypes as C
import os
import shutil
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "computation-suite_b200", "csrc")


COMMON = """#include "feab_common.cuh"
namespace feab {
int sm_count() {
  int d = 0, n = 0;
  cudaGetDevice(&d);
  return cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, d) == cudaSuccess ? n : 1;
}
void count_launches(uint64_t) {}
}
"""


def build(tmp, *sources):
    """A ctypes library of these sources of csrc, or None without nvcc.  Its state (cached graphs) is its own
    beside libfeab200's in the process: no unique symbols, its own definitions first."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        return None
    lib, common = os.path.join(str(tmp), "waits.so"), os.path.join(str(tmp), "common.cu")
    with open(common, "w") as fh:
        fh.write(COMMON)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "--expt-relaxed-constexpr", "-DFEAB_WAIT_CYCLES=0", "-I", os.path.join(ROOT, "include"),
                    "-I", CSRC, "-o", lib, common, *[os.path.join(CSRC, s) for s in sources], "-cudart",
                    "static", "--threads", "4", "-Xcompiler",
                    "-fno-gnu-unique", "-Xlinker", "-Bsymbolic"], check=True, capture_output=True)
    return C.CDLL(lib)
