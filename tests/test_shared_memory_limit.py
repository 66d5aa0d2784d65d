"""The kernels' shared-memory limits are raised on every device that runs them: the helper compiled against stand-ins for the two CUDA
calls that it makes."""

import os
import subprocess

from stride_b200.csrc import build

PROGRAM = r"""
#include "shared_limit.hpp"
#include <cstdio>
static int device = 0, calls[4] = {}, refuse = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, enum cudaFuncAttribute, int bytes) {
    if (refuse) return cudaErrorInvalidValue;
    ++calls[device];
    return bytes == 1000 ? cudaSuccess : cudaErrorInvalidValue;
}
void kernel_a(int) {}
void kernel_b(int) {}
int main() {
    int bad = 0;
    for (int turn = 0; turn < 2; ++turn)
        for (device = 0; device < 3; ++device) bad += stride::allow_shared<kernel_a>(1000) != cudaSuccess;
    bad += calls[0] != 1 || calls[1] != 1 || calls[2] != 1;
    device = 1;
    refuse = 1;
    bad += stride::allow_shared<kernel_b>(1000) == cudaSuccess;       // a refusal is not remembered as done
    refuse = 0;
    bad += stride::allow_shared<kernel_b>(1000) != cudaSuccess || calls[1] != 2;
    device = 64;
    bad += stride::allow_shared<kernel_b>(1000) == cudaSuccess;
    std::printf("%d\n", bad);
    return bad;
}
"""


def test_limits_are_raised_once_a_device(tmp_path):
    include = os.path.join(os.path.dirname(os.path.dirname(build.find_nvcc())), "include")
    source, program = tmp_path / "limit.cpp", tmp_path / "limit"
    source.write_text(PROGRAM)
    made = subprocess.run([build.find_cxx(), "-std=c++17", "-I", build.KERNEL_DIR, "-I", include, str(source), "-o", str(program)],
                          capture_output=True, text=True)
    assert made.returncode == 0, made.stderr
    assert subprocess.run([str(program)], capture_output=True).returncode == 0
