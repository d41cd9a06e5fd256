"""When path-traced frames of a two-level scene build its 4-wide trees, seen in
the handle's device memory: once their bounce segments pay for it, and never in
counted frames. The film is the counted render's, frame by frame, with and
without the trees."""

from __future__ import annotations

import numpy as np
import pytest

from raycer_gb300 import scenes
from raycer_gb300.tracer import CudaTracer, TracerState

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth,builds_at", [(1, None), (2, 4), (3, 2), (4, 2), (5, 1), (9, 1)])
def test_frames_build_the_trees_once_they_pay_for_them(depth, builds_at):
    sc = scenes.heightfield_blobs_instanced(instances=12, blob_level=2, hf_nx=64, hf_nz=32, width=96, height=54,
                                            dielectric_fraction=0.4)
    sc.settings["max_path_length"] = depth
    state = TracerState(scene=sc, filmWidth=sc.width, filmHeight=sc.height, pixelCount=sc.width * sc.height)
    with CudaTracer(0) as t, CudaTracer(0) as ref:
        for tracer in (t, ref):
            tracer.initializeInstanced(sc, seed=3)
            tracer.initializeImageBuffers(sc.width, sc.height)
            tracer.set_counting(True)
        t.run(state)  # the call's buffers
        before = t.stats()["device_bytes"]
        t.clear()
        t.set_counting(False)
        for frame in range(1, 6):
            t.run(state)
            ref.run(state)
            assert np.array_equal(t.read_film(), ref.read_film())
            assert t.stats()["rays_traced"] == ref.stats()["rays_traced"]
            built = t.stats()["device_bytes"] > before
            assert built == (builds_at is not None and frame >= builds_at)
        t.initializeInstanced(sc, seed=3)  # a new upload starts anew
        t.run(state)
        assert (t.stats()["device_bytes"] > before) == (builds_at == 1)
