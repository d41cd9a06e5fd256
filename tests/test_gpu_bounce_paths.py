"""Passes at the sizes where the path tracer's work distribution changes: a
group of 32, 16, 8 or 4 lanes per path (small passes, one kernel), one path
per lane (camera rays, then all later segments in one launch), partial warps;
one segment (no bounce launch), two, and many, with and without Russian
roulette. Films equal the float32 oracle's bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from raycer_gb300.tracer import CudaTracer, TracerState, camera_record

from helpers import camera_floats, small_room

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height,depth,rr", [(2, 2, 4, 0), (3, 11, 2, 0), (3, 11, 1, 0), (62, 89, 6, 3),
                                                   (97, 113, 12, 2), (139, 141, 5, 0), (200, 195, 4, 3),
                                                   (400, 390, 1, 0), (400, 390, 2, 0), (400, 390, 7, 3)])
def test_film_matches_oracle(width, height, depth, rr):
    sc = small_room(width=width, height=height)
    sc.settings.update(multi_sample_count_sqrt=1, path_sample_count=1, max_path_length=depth,
                       russian_roulette_depth=rr)
    n = width * height
    with CudaTracer(0) as t:
        t.initializeBuffers(sc, seed=21)
        t.initializeImageBuffers(width, height)
        st = TracerState(scene=sc, filmWidth=width, filmHeight=height, pixelCount=n)
        t.run(st)
        film = t.read_film()
        rays = t.stats()["rays_traced"]
        cam = camera_floats(camera_record(sc))
    ref, stats = oracle.Oracle(sc).render_path32(cam, width, n, 1, 1, 4, (0.5, 0.5), 1e-5, depth, rr, 1, 21, 0)
    assert np.array_equal(film, ref), f"{(film != ref).any(axis=1).sum()} pixels differ"
    assert n <= rays <= n * depth
