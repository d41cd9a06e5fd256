"""Calls with few rays walk each ray with a group of 32, 16, 8 or 4 lanes
(traverse_group); the group follows from the number of rays. Larger casts walk
one ray per lane in warp-wide phases. Casts and RAY
frames on both sides of every line, and with a partial last warp, equal the
float32 oracle's bit for bit in both orders, as do overlapping coplanar
triangles (where box rounding decides ties) and rays with NaN components."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from raycer_gb300 import _native as N
from raycer_gb300.tracer import CudaTracer, TracerState, camera_record

from helpers import camera_floats, small_heightfield, small_room
from test_gpu_degenerate import scene as degenerate_scene

pytestmark = pytest.mark.gpu

ORDERS = [N.RC_ORDER_REFERENCE, N.RC_ORDER_NEAREST]


def _rays(n, seed, nan_every=0):
    rng = np.random.default_rng(seed)
    rays = np.zeros(n, dtype=[("origin", "<f4", 3), ("t_min", "<f4"), ("direction", "<f4", 3), ("t_max", "<f4")])
    rays["origin"] = rng.uniform(-0.95, 0.95, size=(n, 3))
    d = rng.normal(size=(n, 3))
    rays["direction"] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays["t_max"] = np.where(rng.uniform(size=n) < 0.5, np.float32(3.0e38), rng.uniform(0.1, 2.0, size=n))
    if nan_every:
        rays["direction"][::nan_every, 1] = np.nan
    return rays


@pytest.mark.parametrize("n", [1, 3, 33, 19_457, 38_917, 77_833, 311_299, 311_400])
@pytest.mark.parametrize("order", ORDERS)
def test_casts(n, order):
    sc = small_room(clutter=1000)
    rays = _rays(n, n, nan_every=7 if n < 100 else 0)
    orc = oracle.Oracle(sc)
    with CudaTracer(0) as t:
        t.initializeBuffers(sc)
        for any_hit in (False, True):
            hits = t.cast(rays, any_hit=any_hit, order=order)
            prim, tt, u, v, _ = orc.cast32(rays, any_hit=any_hit, order=order)
            assert np.array_equal(hits["prim"], prim)
            for k, ref in (("t", tt), ("u", u), ("v", v)):
                assert np.array_equal(hits[k], ref, equal_nan=True)


@pytest.mark.parametrize("width,height", [(2, 2), (13, 9), (100, 97), (139, 140), (277, 141), (401, 389)])
@pytest.mark.parametrize("order", ORDERS)
def test_frames(width, height, order):
    sc = small_heightfield(width=width, height=height)
    sc.light_direction = (-1.0, -0.25, -0.2)
    n = width * height
    with CudaTracer(0) as t:
        t.initializeBuffers(sc)
        t.set_traversal_order(order)
        t.initializeImageBuffers(width, height)
        st = TracerState(scene=sc, filmWidth=width, filmHeight=height, pixelCount=n)
        t.run(st)
        assert st.pixelsProcessed == n
        got = t.read_cast().view(np.int32).reshape(-1, 4)
        part = n // 3 + 1
        t.clear()
        t.run(TracerState(scene=sc, filmWidth=width, filmHeight=height, pixelStartOffset=n - part, pixelCount=part))
        tail = t.read_cast().view(np.int32).reshape(-1, 4)[:part]
        cam = camera_floats(camera_record(sc))
    ref, _ = oracle.Oracle(sc).raycast32(cam, width, n, -np.array(sc.light_direction, np.float32), order=order)
    assert np.array_equal(got, ref)
    assert np.array_equal(tail, ref[n - part:])


@pytest.mark.parametrize("n", [500, 30_000, 330_000])
@pytest.mark.parametrize("order", ORDERS)
def test_coplanar(n, order):
    sc = degenerate_scene("coplanar", 4)
    rays = _rays(n, 5)
    with CudaTracer(0) as t:
        t.initializeBuffers(sc)
        hits = t.cast(rays, order=order)
    prim, tt, _, _, _ = oracle.Oracle(sc).cast32(rays, any_hit=False, order=order)
    assert np.array_equal(hits["prim"], prim)
    assert np.array_equal(hits["t"], tt)
