"""The progress that rc_render reports while a RAY frame runs never passes the
pixels it has finished: read by another thread until the frame's time budget
stops it, it stays within the exact count that the call returns. The films are
narrower than two 8-pixel tiles, so most of the tiles' pixels lie outside."""

from __future__ import annotations

import threading

import pytest

from raycer_gb300 import _native as N
from raycer_gb300.tracer import CudaTracer, RaycerError, TracerState

from helpers import small_heightfield

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", [0, 5])
@pytest.mark.parametrize("order", [N.RC_ORDER_NEAREST, N.RC_ORDER_REFERENCE])
def test_progress_stays_within_the_finished_pixels(order, first):
    width, height = 9, 4_000_000
    sc = small_heightfield(width=width, height=height)
    sc.settings["tracer"] = "ray"
    with CudaTracer(0) as t:
        t.initializeBuffers(sc)
        t.set_traversal_order(order)
        t.initializeImageBuffers(width, height)
        n = width * height - first
        state = TracerState(scene=sc, filmWidth=width, filmHeight=height, pixelStartOffset=first, pixelCount=n)
        t.run(state)
        whole = t.stats()["last_ms"]
        t.set_time_budget(0.6 * whole)
        for _ in range(5):
            seen = [0]
            done = threading.Event()

            def watch():
                while not done.is_set():
                    seen.append(state.pixelsProcessed)

            state.pixelsProcessed = 0
            reader = threading.Thread(target=watch)
            reader.start()
            with pytest.raises(RaycerError) as stopped:
                t.run(state)
            done.set()
            reader.join()
            assert stopped.value.status == N.RC_TIMEOUT
            assert 0 < state.pixelsProcessed < n
            assert all(a <= b for a, b in zip(seen, seen[1:]))
            assert max(seen) <= state.pixelsProcessed
