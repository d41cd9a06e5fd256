"""RAY frames of pixel ranges in tiles on the film's columns: a range's records
are the whole frame's, pixel by pixel. Ranges that start and end within a line
and within a tile, films whose lines are no whole tiles, ranges of just four
lines and of one pixel less (in order), on both sides of the size where a ray
gets a group of lanes; both traversal orders."""

from __future__ import annotations

import numpy as np
import pytest

from raycer_gb300 import scenes
from raycer_gb300 import _native as N
from raycer_gb300.tracer import CudaTracer, TracerState

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [N.RC_ORDER_NEAREST, N.RC_ORDER_REFERENCE])
@pytest.mark.parametrize("width,height,ranges", [
    (613, 397, [(0, 613 * 397), (5, 200003), (613 * 7 + 612, 180001), (100, 4 * 613), (100, 4 * 613 - 1)]),
    (640, 400, [(0, 640 * 300), (639, 170001), (640 * 3, 640 * 397)]),
    (9, 25001, [(4, 9 * 25001 - 9), (0, 37)]), (7, 30001, [(3, 7 * 30001 - 5)])])
def test_range_is_the_frames(width, height, ranges, order):
    sc = scenes.heightfield_scene(nx=96, nz=48)
    sc.width, sc.height = width, height
    with CudaTracer(0) as t:
        t.initializeBuffers(sc)
        t.initializeImageBuffers(width, height)
        t.set_traversal_order(order)
        n = width * height
        t.run(TracerState(scene=sc, filmWidth=width, filmHeight=height, pixelCount=n))
        frame = t.read_cast().copy()
        assert (frame["prim"] >= 0).any()
        for first, count in ranges:
            t.run(TracerState(scene=sc, filmWidth=width, filmHeight=height, pixelStartOffset=first, pixelCount=count))
            part = t.read_cast()[:count]
            assert part.tobytes() == frame[first:first + count].tobytes(), (first, count)
