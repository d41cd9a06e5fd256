"""Frames, casts and passes around the sizes where groups of 32, 16, 8 and 4
lanes per ray give way to each other and to one ray per lane, which depend on
the scene's size: results equal the float32 oracle's bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from raycer_gb300 import _native as N
from raycer_gb300 import scenes
from raycer_gb300.tracer import CudaTracer, TracerState, camera_record

from helpers import camera_floats

pytestmark = pytest.mark.gpu

# a group of 4 lanes for each of this many rays fills a GB300's resident warps
LANES = 152 * 8 * 128 // 4


@pytest.mark.parametrize("nx,nz", [(2, 2), (12, 8), (96, 48), (240, 120)])
@pytest.mark.parametrize("share", [0.03, 0.12, 0.24, 0.26, 0.49, 0.51, 0.97, 1.03, 1.3])
@pytest.mark.parametrize("order", [N.RC_ORDER_REFERENCE, N.RC_ORDER_NEAREST])
def test_frames(nx, nz, share, order):
    width = 211
    height = max(2, int(share * LANES) // width)
    sc = scenes.heightfield_scene(nx=nx, nz=nz, width=width, height=height)
    sc.settings["tracer"] = "ray"
    sc.light_direction = (-1.0, -0.25, -0.2)
    n = width * height
    with CudaTracer(0) as t:
        t.initializeBuffers(sc)
        t.set_traversal_order(order)
        t.initializeImageBuffers(width, height)
        t.run(TracerState(scene=sc, filmWidth=width, filmHeight=height, pixelCount=n))
        got = t.read_cast().view(np.int32).reshape(-1, 4)
        cam = camera_floats(camera_record(sc))
    ref, _ = oracle.Oracle(sc).raycast32(cam, width, n, -np.array(sc.light_direction, np.float32), order=order)
    assert np.array_equal(got, ref), f"{(got != ref).any(axis=1).sum()} pixels differ"
