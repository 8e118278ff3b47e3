"""The object dependencies of the CUDA library's build: a changed header rebuilds
the objects that include it, a removed one does not stop the build."""

from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

MAKEFILE = Path(__file__).resolve().parents[1] / "witwin_channel_b200" / "csrc" / "Makefile"


@pytest.mark.skipif(shutil.which("nvcc") is None or shutil.which("make") is None, reason="needs nvcc and make")
def test_headers_may_change_and_go(tmp_path):
    shutil.copy(MAKEFILE, tmp_path / "Makefile")

    def make():
        return subprocess.run(["make", "a.o", "SRCS=a.cu"], cwd=tmp_path, capture_output=True, text=True)

    (tmp_path / "b.cuh").write_text("constexpr int kValue = 1;\n")
    (tmp_path / "a.cu").write_text('#include "b.cuh"\nint value() { return kValue; }\n')
    assert make().returncode == 0
    assert "up to date" in make().stdout
    (tmp_path / "b.cuh").write_text("constexpr long kValue = 2;\n")
    assert "-c a.cu" in make().stdout
    (tmp_path / "b.cuh").unlink()
    (tmp_path / "a.cu").write_text("int value() { return 3; }\n")
    out = make()
    assert out.returncode == 0, out.stderr
    assert "-c a.cu" in out.stdout
