"""The shared-memory limit of a kernel belongs to one device: it is raised once on each, never once per process.  Checked on the CPU against a
CUDA runtime of two functions."""
import glob
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "my_nn_engine_b200", "csrc")

PROGRAM = r"""
#include <stdio.h>
#include "smem_limit.h"
static int device, calls, refuse;
extern "C" cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void *, enum cudaFuncAttribute a, int bytes) {
    if (refuse) return cudaErrorInvalidValue;
    calls += a == cudaFuncAttributeMaxDynamicSharedMemorySize && bytes == 100000;
    return cudaSuccess;
}
int main() {
    mynn::SmemLimit one, two;
    char kern;
    auto on = [&](mynn::SmemLimit &l, int d) { device = d; return l.raise(&kern, 100000); };
    refuse = 1;
    printf("%d ", on(one, 0) != cudaSuccess);  // a failure is reported and tried again
    refuse = 0;
    on(one, 0), on(one, 0); printf("%d ", calls);
    on(one, 1), on(one, 1), on(one, 0); printf("%d ", calls);
    on(two, 0), on(two, 63), on(two, 63); printf("%d ", calls);
    on(two, 64), on(two, 64); printf("%d\n", calls);
}
"""


def test_limit_is_raised_once_per_device(tmp_path):
    (tmp_path / "p.cpp").write_text(PROGRAM)
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-I", cuda, str(tmp_path / "p.cpp"), "-o", str(tmp_path / "p")], check=True)
    out = subprocess.run([str(tmp_path / "p")], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["1", "1", "2", "4", "6"]


def test_no_launcher_remembers_it_for_the_whole_process():
    """A limit is set on every launch that needs it, or through SmemLimit."""
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        lines = open(path).read().split("\n")
        for i, line in enumerate(lines):
            if "cudaFuncAttributeMaxDynamicSharedMemorySize" in line:
                assert not any("static bool" in before for before in lines[max(0, i - 4):i]), f"{path}:{i + 1}"
