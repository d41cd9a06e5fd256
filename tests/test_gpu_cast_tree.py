"""When rc_cast builds the scene's 4-wide tree, seen in the handle's device
memory: once the rays pay for it, and never where its kernels would not walk it
(the stackless switch). Casts through a tree that is there equal the float32
oracle's at the sizes where the kernels change."""

from __future__ import annotations

import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import oracle
from raycer_gb300 import _native as N
from raycer_gb300.tracer import RAY_DTYPE, CudaTracer, camera_record

from helpers import camera_floats, small_heightfield, small_room
from test_gpu_degenerate import scene as degenerate_scene
from test_gpu_ray_groups import _rays

pytestmark = pytest.mark.gpu

TESTS = Path(__file__).resolve().parent


def grow_tree(t):
    """Has the tracer's scene build its 4-wide tree: a cast of many empty rays."""
    rays = np.zeros(4_000_000, RAY_DTYPE)
    rays["direction"][:, 2] = 1.0
    rays["t_max"] = -1.0
    t.cast(rays, any_hit=True)  # the call's buffers
    before = t.stats()["device_bytes"]
    t.cast(rays)
    t.cast(rays)
    return t.stats()["device_bytes"] - before


def test_casts_build_the_tree_once_they_pay_for_it():
    sc = small_heightfield()
    rays = _rays(2_100_000, 3)
    with CudaTracer(0) as t:
        for _ in range(2):  # the second upload starts anew
            t.initializeBuffers(sc)
            t.cast(rays, any_hit=True)
            before = t.stats()["device_bytes"]
            grown = []
            first = t.cast(rays)
            for _ in range(4):
                grown.append(t.stats()["device_bytes"] - before)
                assert np.array_equal(t.cast(rays), first)
            t.cast(rays[:300_000])
            t.cast(rays, order=N.RC_ORDER_REFERENCE)
            assert grown[0] == grown[1] == grown[2] == 0 and grown[3] > 0
            assert grown[3] == t.stats()["device_bytes"] - before
        t.initializeBuffers(sc)
        assert grow_tree(t) == grown[3]


@pytest.mark.parametrize("n", [1_245_184, 1_245_185, 1_300_000])
@pytest.mark.parametrize("name", ["room", "terrain", "coplanar", "duplicates"])
def test_casts_through_the_tree(name, n):
    sc = {"room": lambda: small_room(clutter=1000), "terrain": small_heightfield,
          "coplanar": lambda: degenerate_scene("coplanar", 4), "duplicates": lambda: degenerate_scene("duplicates", 1)}[name]()
    rays = _rays(n, n)
    with CudaTracer(0) as t:
        t.initializeBuffers(sc)
        assert grow_tree(t) > 0
        hits = t.cast(rays)
    prim, tt, u, v, _ = oracle.Oracle(sc).cast32(rays, any_hit=False, order=N.RC_ORDER_NEAREST)
    assert np.array_equal(hits["prim"], prim)
    for k, ref in (("t", tt), ("u", u), ("v", v)):
        assert np.array_equal(hits[k], ref)


@pytest.mark.parametrize("frame", [1.0, 0.55, 0.45])
def test_large_casts_of_a_frames_rays(frame):
    """Rays that walk together, and batches of which about half do."""
    width, height = 1400, 1000
    sc = small_heightfield(width=width, height=height)
    n = width * height
    rays = _rays(n, 9)
    cam = np.ascontiguousarray(oracle.camera_rays32(camera_floats(camera_record(sc)), width, n))
    first = int(frame * n)
    rays[:first] = cam.view(rays.dtype).reshape(-1)[:first]
    orc = oracle.Oracle(sc)
    with CudaTracer(0) as t:
        t.initializeBuffers(sc)
        assert grow_tree(t) > 0
        for any_hit, order in ((False, N.RC_ORDER_NEAREST), (False, N.RC_ORDER_REFERENCE), (True, N.RC_ORDER_NEAREST)):
            hits = t.cast(rays, any_hit=any_hit, order=order)
            prim, tt, u, v, _ = orc.cast32(rays, any_hit=any_hit, order=order)
            assert np.array_equal(hits["prim"], prim)
            for k, ref in (("t", tt), ("u", u), ("v", v)):
                assert np.array_equal(hits[k], ref)
            assert t.stats()["rays_traced"] == n


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
