"""The opt-in to large dynamic shared memory holds on every device that a process uses."""
import glob
import os
import re

from rockseis_b200 import build
from tests.host_cc import run_cpp

FAKE = r"""
#include <cstdio>
#include "smem_limit.h"
static int device = 0, calls[80] = {}, fail = 0;
extern "C" cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int bytes)
{
    calls[device] += bytes == 70000;
    return fail ? cudaErrorInvalidValue : cudaSuccess;
}
static void kernel(int) {}
int main()
{
    rsgpu::SmemLimit l;
    for (int round = 0; round < 3; round++)
        for (device = 0; device < 4; device++)
            if (l.raise(kernel, 70000) != cudaSuccess) return 1;
    for (int d = 0; d < 4; d++) printf("%d ", calls[d]);
    // a refusal is reported and not remembered
    device = 5; fail = 1;
    if (l.raise(kernel, 70000) == cudaSuccess) return 2;
    fail = 0;
    if (l.raise(kernel, 70000) != cudaSuccess || l.raise(kernel, 70000) != cudaSuccess) return 3;
    device = 70;
    for (int k = 0; k < 2; k++) if (l.raise(kernel, 70000) != cudaSuccess) return 4;
    printf("%d %d\n", calls[5], calls[70]);
}
"""


def test_raised_once_on_each_device(tmp_path):
    assert run_cpp(tmp_path, FAKE).split() == ["1", "1", "1", "1", "2", "2"]


def test_no_launcher_raises_it_once_per_process():
    # fd2d_fused.cu and fd2d_march.cu also raise it on the plan's device when a plan is created
    for path in glob.glob(os.path.join(build.CSRC, "*.cu*")):
        if os.path.basename(path) in ("fd2d_fused.cu", "fd2d_march.cu"):
            continue
        with open(path) as f:
            assert not re.search(r"static\s+(const\s+)?cudaError_t\s+\w+\s*=", f.read()), path
