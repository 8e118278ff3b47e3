"""The FP32 Fresnel sum at arguments far past the range of ordinary links (an
endpoint within a fraction of a millimetre of an edge), compiled for the
host.  |(1+j)/2 - (C + jS)(x)| -> 1 / (pi x) with a next term of 3 / (pi^2 x^4)
relative; its two factors, the product and the modulus round by 2^-24 each:
1e-6.  The share of an edge end that the stationary point lies beyond is the
same modulus over sqrt 2 on the near side and (its real plus imaginary part) / 2
on the far side, whose phase pi x^2 / 2 reduced in FP64 is off by 2^-53 of
itself: 1e-6 of the modulus up to x = 1e4, checked there against the FP64
evaluation of the same functions; the modulus is checked to 1e9."""

from __future__ import annotations

import shutil
import subprocess

import numpy as np
import pytest

from tests.test_utd_special_cpu import CSRC, CUDA_INCLUDE

PROGRAM = r"""
#include <cmath>
#include <cstdio>
using std::isfinite;
#include "utd.cuh"
using namespace wcb;

int main() {
    for (int i = 0; i < 2000; ++i) {
        const float x = float(std::pow(10.0, 2.0 + 7.0 * i / 1999.0));
        const Cx<float> c = fresnel_pos<float>(x).complement(x, fresnel_phasor<float>(double(x)));
        const double m = std::hypot(double(c.re), double(c.im));
        std::printf("%.9g %.17g %.9g %.9g %.17g %.17g\n", x, m, fresnel_end_share<float>(double(x)),
                    fresnel_end_share<float>(-double(x)), fresnel_end_share<double>(double(x)),
                    fresnel_end_share<double>(-double(x)));
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def values(tmp_path_factory):
    if shutil.which("g++") is None or not (CUDA_INCLUDE / "cuda_runtime.h").exists():
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("far")
    (d / "main.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-w", "-D__noinline__=", f"-I{CUDA_INCLUDE}", f"-I{CSRC}",
                    str(d / "main.cpp"), "-o", str(d / "main")], check=True)
    out = subprocess.run([str(d / "main")], check=True, capture_output=True, text=True).stdout
    return np.array([[float(t) for t in line.split()] for line in out.splitlines()])


def test_complement_modulus(values):
    x, m = values[:, 0], values[:, 1]
    assert np.all(np.abs(m * np.pi * x - 1.0) <= 1e-6)


def test_end_share(values):
    x, near, far, near64, far64 = values[:, 0], values[:, 2], values[:, 3], values[:, 4], values[:, 5]
    assert np.all(np.abs(near - near64) <= 1e-6 * near64)
    ok = x <= 1e4
    assert np.all(np.abs(far - far64)[ok] <= (1e-6 / (np.pi * x))[ok])
    # past it the share still has the size of the complement
    assert np.max((np.abs(far) * np.pi * x)[~ok]) <= 1.0
    assert np.max((np.abs(far) * np.pi * x)[x > 1e8]) >= 0.5
