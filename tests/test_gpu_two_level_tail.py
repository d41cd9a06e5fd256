"""The last paths of a two-level frame: a warp whose queue has run dry and whose
remaining lanes are all on their way out of an instance still finishes them.
Frames over 50 small meshes, where that happens a few times per frame, equal
the counted renders' films bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

from raycer_gb300 import scenes
from raycer_gb300.tracer import CudaTracer, TracerState

pytestmark = pytest.mark.gpu


def _films(sc, seed, counting, frames):
    out = []
    with CudaTracer(0) as t:
        t.initializeInstanced(sc, seed=seed)
        t.initializeImageBuffers(sc.width, sc.height)
        t.set_counting(counting)
        for _ in range(frames):
            t.run(TracerState(scene=sc, filmWidth=sc.width, filmHeight=sc.height, pixelCount=sc.width * sc.height))
            out.append(t.read_film().copy())
    return out


@pytest.mark.parametrize("seed", [1, 2, 3, 4])
def test_films_of_many_small_meshes(seed):
    sc = scenes.heightfield_blobs_instanced(instances=50, blob_level=2, hf_nx=150, hf_nz=322, width=522, height=414,
                                            dielectric_fraction=0.22)
    sc.settings["max_path_length"] = 5
    for k, (film, ref) in enumerate(zip(_films(sc, seed, False, 8), _films(sc, seed, True, 8))):
        assert np.array_equal(film, ref), f"frame {k}: {(film != ref).any(axis=1).sum()} pixels differ"
