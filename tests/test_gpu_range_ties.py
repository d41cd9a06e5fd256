"""RAY frames of pixel ranges among overlapping triangles of common planes,
where the order of a walk can decide between hits that rounding puts before
their boxes: the records are the float32 oracle's, whose order is the ray's
own, on both sides of the line where groups of lanes end."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from raycer_gb300 import _native as N
from raycer_gb300 import scenes
from raycer_gb300.tracer import CudaTracer, TracerState, camera_record

from helpers import camera_floats
from test_gpu_two_level_ties import _sheet

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first,count", [(301, 288_360), (8010, 320_400), (0, 480_599), (5, 100_000)])
@pytest.mark.parametrize("order", [N.RC_ORDER_NEAREST, N.RC_ORDER_REFERENCE])
def test_ranges_in_a_room_of_sheets(order, first, count):
    width, height = 801, 600
    rng = np.random.default_rng(8)
    v = np.concatenate([_sheet(rng, 60, axis, s, 1.2, 0.5) for axis in range(3) for s in (-1.3, 1.3)])
    sc = scenes.SceneDesc("room", v, np.zeros(len(v), np.uint32), [scenes.Material(diffuse=(0.6, 0.6, 0.6))],
                          scenes.CameraDesc(position=(0.05, 0.1, 4.0), fov=50.0), width, height,
                          light_direction=(-0.4, -1.0, -0.6), max_leaf_size=4, settings={"tracer": "ray"})
    with CudaTracer(0) as t:
        t.initializeBuffers(sc)
        t.set_traversal_order(order)
        t.initializeImageBuffers(width, height)
        t.run(TracerState(scene=sc, filmWidth=width, filmHeight=height, pixelStartOffset=first, pixelCount=count))
        got = t.read_cast().view(np.int32).reshape(-1, 4)[:count]
        cam = camera_floats(camera_record(sc))
    ref, _ = oracle.Oracle(sc).raycast32(cam, width, count, -np.array(sc.light_direction, np.float32), order=order,
                                         pixel_start=first)
    assert np.array_equal(got, ref), f"{(got != ref).any(axis=1).sum()} pixels differ"
