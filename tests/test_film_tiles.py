"""The tiles in which pixel ranges are taken (film_tiles), checked on the host
(film_tiles_check.cpp): films of 2^30 pixels and more are taken in tiles as
smaller ones are; the pixels of a number of tiles."""

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
def test_film_tiles(tmp_path):
    exe = tmp_path / "film_tiles_check"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{_cuda_home() / 'include'}",
                    str(ROOT / "tests" / "film_tiles_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    assert "film tiles ok" in out.stdout
