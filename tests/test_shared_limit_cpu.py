"""The kernels' dynamic shared memory limit is raised on every device that a
process uses, once each, and tried again after a failure; the launch header
compiled for the host with stand-ins for the two runtime calls."""

from __future__ import annotations

import shutil
import subprocess

import pytest

from tests.test_utd_special_cpu import CSRC, CUDA_INCLUDE

PROGRAM = r"""
#include <cmath>
#include <cstdio>
using std::isfinite;
#include "launch.h"

static int device = 0, fail = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int bytes) {
    std::printf("%d:%d%s ", device, bytes, fail ? "!" : "");
    return fail ? cudaErrorInvalidValue : cudaSuccess;
}

int main() {
    static std::atomic<unsigned long long> done{0};
    const int devices[] = {0, 0, 1, 1, 0, 7, 1};
    for (int d : devices) {
        device = d;
        wcb::raise_shared_limit(nullptr, 1024, done);
    }
    device = 3;
    fail = 1;
    wcb::raise_shared_limit(nullptr, 1024, done);
    fail = 0;
    wcb::raise_shared_limit(nullptr, 1024, done);
    wcb::raise_shared_limit(nullptr, 1024, done);
    return 0;
}
"""


def test_once_per_device(tmp_path):
    if shutil.which("g++") is None or not (CUDA_INCLUDE / "cuda_runtime.h").exists():
        pytest.skip("needs g++ and the CUDA headers")
    (tmp_path / "main.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-w", "-D__noinline__=", f"-I{CUDA_INCLUDE}", f"-I{CSRC}",
                    str(tmp_path / "main.cpp"), "-o", str(tmp_path / "main")], check=True)
    out = subprocess.run([str(tmp_path / "main")], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["0:1024", "1:1024", "7:1024", "3:1024!", "3:1024"]


def test_no_kernel_keeps_the_limit_of_one_device():
    text = (CSRC / "launch_components.cuh").read_text()
    assert "static bool" not in text and "cudaFuncSetAttribute" not in text
