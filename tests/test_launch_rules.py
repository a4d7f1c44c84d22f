"""What the host code does when a launch is refused, on the CPU: a source of the library is compiled into a
program that replaces the CUDA calls by ones that answer as a part of a device would."""
import os
import shutil
import subprocess

import pytest
from conftest import ROOT

CSRC = os.path.join(ROOT, "computation-suite_b200", "csrc")
FAKES = """
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <vector>
namespace feab {
int sm_count() { return 148; }
uint64_t launches = 0;
void count_launches(uint64_t n) { launches += n; }
}
static unsigned sms_at_hand = 148;
static bool clusters = true;
static std::vector<unsigned> grids;
static cudaError_t fake_cooperative(const void*, dim3 g, dim3, void**, size_t, cudaStream_t) {
  grids.push_back(g.x);
  return g.x > sms_at_hand ? cudaErrorCooperativeLaunchTooLarge : cudaSuccess;
}
static cudaError_t fake_ex(const cudaLaunchConfig_t* c, const void*, void**) {
  grids.push_back(c->gridDim.x);
  return clusters ? cudaSuccess : cudaErrorInvalidClusterSize;
}
#define cudaLaunchCooperativeKernel fake_cooperative
#define cudaLaunchKernelExC fake_ex
#define cudaFuncSetAttribute(...) cudaSuccess
#define cudaMemcpyAsync(...) cudaSuccess
#define cudaMemsetAsync(...) cudaSuccess
#define cudaStreamSynchronize(...) cudaSuccess
#define cudaGetLastError() cudaSuccess
#define cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, ...) (*(n) = 1, cudaSuccess)
"""


def _run(tmp_path, source, main, *flags):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    src, exe = str(tmp_path / "t.cu"), str(tmp_path / "t")
    with open(src, "w") as fh:
        fh.write(FAKES + f'#include "{source}"\n' + main)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=compute_100a", "-std=c++17", "--expt-relaxed-constexpr",
                    "-I", os.path.join(ROOT, "include"), "-I", CSRC, *flags, src, "-o", exe], check=True, capture_output=True)
    # no device is visible: a launch that is not replaced ends on the host
    out = subprocess.run([exe], check=True, capture_output=True, text=True, env=dict(os.environ, CUDA_VISIBLE_DEVICES=""))
    return [[int(v) for v in line.split()] for line in out.stdout.splitlines()]


def test_band_factor_and_solve_on_a_part_of_a_device(tmp_path):
    out = _run(tmp_path, "feab_band.cu", """
    int main() {
      void* storage = aligned_alloc(256, 1 << 20);
      double *b = (double*)storage + 1, *x = b + 1, *w = x + 1;
      int32_t flag = 0;
      for (int bands : {0, 5, 20, 200}) {
        feab_band B{64 * 300, 300, bands, 0, storage};
        for (unsigned sms : {148u, 40u, 2u, 1u}) {
          sms_at_hand = sms;
          grids.clear();
          printf("%d ", feab_band_cholesky(&B, nullptr, nullptr));
          for (unsigned g : grids) printf("%u ", g);
          printf("\\n");
        }
        for (bool c : {true, false}) {
          clusters = c;
          grids.clear();
          feab::launches = 0;
          printf("%d ", feab_band_solve_flag(&B, b, x, w, &flag, nullptr));
          printf("%d %d\\n", (int)grids.size(), (int)feab::launches);
        }
      }
    }
    """)
    CUDA_ERROR = 6
    factor = [[[0, 1]] * 4] + [[[0, 148], [0, 148, 74, 37], [0, 148, 74, 37, 18, 9, 4, 2],
                                [CUDA_ERROR, 148, 74, 37, 18, 9, 4, 2]]] * 3
    for i, bands in enumerate((0, 5, 20, 200)):
        rows = out[6 * i:6 * i + 6]
        assert rows[:4] == factor[i], bands
        # one cluster kernel, and a launch per block row and direction where it is refused or too wide
        assert rows[4] == ([0, 1, 1] if bands <= 128 else [0, 0, 600]), bands
        assert rows[5] == ([0, 1, 600] if bands <= 128 else [0, 0, 600]), bands


@pytest.mark.parametrize("fused", [0, 1])
def test_step_kernel_of_the_sliced_operator(tmp_path, fused):
    """The direction formed inside step A's gathers (a build option) is not one that the ring can take."""
    out = _run(tmp_path, "feab_pcg.cu", """
    int main() {
      using namespace feab;
      char* at = (char*)aligned_alloc(256, 4096);
      for (int off : {0, 2}) {
        PcgArgs A{};
        A.sell.tcol16 = (const int16_t*)(at + off);
        A.sell.v64 = (double*)at;
        A.sell.vhi = (uint32_t*)at;
        A.sell.vlo = (uint16_t*)at;
        printf("%d %d\\n", (int)sell_ring(A, FEAB_PREC_FP64), (int)sell_ring(A, FEAB_PREC_MIXED));
      }
      exit(0);
    }
    """, f"-DFEAB_SELL_FUSED_P={fused}", "-Xlinker", "--unresolved-symbols=ignore-all", "-Xcicc", "-O0")
    assert out == [[1 - fused, 1 - fused], [0, 0]]
