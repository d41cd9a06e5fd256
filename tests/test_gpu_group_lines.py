"""Frames, casts and passes around the sizes where groups of 32, 16, 8 and 4
lanes per ray give way to each other and to one ray per lane, which depend on
the scene's size: results equal the float32 oracle's bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from raycer_gb300 import _native as N
from raycer_gb300 import scenes
from raycer_gb300.tracer import RAY_DTYPE, CudaTracer, TracerState, camera_record

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


@pytest.mark.parametrize("nx,nz", [(2, 2), (12, 8), (30, 26), (96, 48), (150, 120), (300, 151)])
@pytest.mark.parametrize("n", [1, 2_400, 2_500, 9_700, 9_800, 25_900, 26_000, 38_900, 39_000, 68_000, 68_200, 77_900, 155_700])
def test_casts(nx, nz, n):
    sc = scenes.heightfield_scene(nx=nx, nz=nz)
    rng = np.random.default_rng(n)
    v = sc.vertices.reshape(-1, 3)
    rays = np.zeros(n, RAY_DTYPE)
    rays["origin"] = rng.uniform(v.min(0) - 0.1, v.max(0) + 0.1, size=(n, 3))
    rays["direction"] = rng.normal(size=(n, 3))
    rays["t_max"] = np.where(rng.random(n) < 0.5, np.float32(3.0e38), np.float32(2.0))
    orc = oracle.Oracle(sc)
    with CudaTracer(0) as t:
        t.initializeBuffers(sc)
        for any_hit, order in ((False, N.RC_ORDER_NEAREST), (False, N.RC_ORDER_REFERENCE), (True, N.RC_ORDER_NEAREST)):
            hits = t.cast(rays, any_hit=any_hit, order=order)
            prim, tt, u, v_, _ = orc.cast32(rays, any_hit=any_hit, order=order)
            assert np.array_equal(hits["prim"], prim)
            for k, ref in (("t", tt), ("u", u), ("v", v_)):
                assert np.array_equal(hits[k], ref, equal_nan=True)


@pytest.mark.parametrize("nx,nz", [(12, 8), (96, 48), (240, 120)])
@pytest.mark.parametrize("share", [0.015, 0.06, 0.12, 0.24, 0.26, 0.66, 0.68, 0.97, 1.03, 1.32, 1.35])
@pytest.mark.parametrize("depth", [1, 3])
def test_passes(nx, nz, share, depth):
    width = 211
    height = max(2, int(share * LANES) // width)
    sc = scenes.heightfield_path_scene(nx=nx, nz=nz, width=width, height=height, max_path_length=depth)
    n = width * height
    with CudaTracer(0) as t:
        t.initializeBuffers(sc, seed=21)
        t.initializeImageBuffers(width, height)
        t.run(TracerState(scene=sc, filmWidth=width, filmHeight=height, pixelCount=n))
        film = t.read_film()
        cam = camera_floats(camera_record(sc))
    ref, _ = oracle.Oracle(sc).render_path32(cam, width, n, 1, 1, 4, (0.5, 0.5), 1e-5, depth, 0, 1, 21, 0)
    assert np.array_equal(film, ref), f"{(film != ref).any(axis=1).sum()} pixels differ"
