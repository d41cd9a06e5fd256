"""The 4-wide trees' construction (wide_host.cpp, wide_collapse.h) on the host,
against a CUDA runtime whose device is host memory (wide_build_check.cpp, with
the address sanitizer): random trees keep their leaves; the child of largest
area is opened; links that are no tree are reported and never followed; scenes
for whose trees there is no memory stay binary."""

from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def _cuda_home() -> Path | None:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    home = Path(nvcc).resolve().parent.parent
    return home if (home / "include" / "cuda_runtime.h").exists() else None


@pytest.mark.skipif(shutil.which("g++") is None or _cuda_home() is None, reason="no C++ compiler or CUDA headers")
def test_wide_build_on_the_host(tmp_path):
    exe = tmp_path / "wide_build_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address", f"-I{_cuda_home() / 'include'}",
                    str(ROOT / "tests" / "wide_build_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    assert "wide build ok" in out.stdout
