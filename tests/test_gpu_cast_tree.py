"""When rc_cast builds the scene's 4-wide tree, seen in the handle's device
memory: never where its kernels would not walk it (the stackless switch)."""

from __future__ import annotations

import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

TESTS = Path(__file__).resolve().parent

_STACKLESS = """
import sys
sys.path.insert(0, {root!r})
sys.path.insert(0, {tests!r})
from helpers import small_room
from raycer_gb300.tracer import CudaTracer
from test_gpu_ray_groups import _rays

rays = _rays(400_000, 3)
with CudaTracer(0) as t:
    t.initializeBuffers(small_room(clutter=1000))
    t.cast(rays, any_hit=True)
    before = t.stats()["device_bytes"]
    for _ in range(12):
        t.cast(rays)
    assert t.stats()["device_bytes"] == before, (before, t.stats()["device_bytes"])
print("no tree")
"""


def test_stackless_casts_build_no_tree():
    env = dict(os.environ, RC_STACKLESS="1")
    out = subprocess.run([sys.executable, "-c", _STACKLESS.format(root=str(TESTS.parent), tests=str(TESTS))], env=env,
                         capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    assert "no tree" in out.stdout
