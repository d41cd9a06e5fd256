"""Camera rays made by the kernel that traces them and taken in 8x4-pixel tiles,
against the counted render, which generates them apart and in slot order: films
and radiance-cache training records are the same. Sizes: tiles cut off at the
right and the bottom, a rest of less than a line, fewer than four lines (no
tiles), a range that starts and ends within a line, several samples per pixel,
a last training run whose path lies past the pass; small passes (groups of
lanes), large ones, and two-level scenes."""

from __future__ import annotations

import numpy as np
import pytest

from raycer_gb300.nrc import RadianceCache
from raycer_gb300.scenes import heightfield_blobs_instanced
from raycer_gb300.tracer import CudaTracer, TracerState

from helpers import nrc_init_params, small_room

pytestmark = pytest.mark.gpu


def _render(sc, width, height, first, count, counting, cache, instanced):
    with CudaTracer(0) as t:
        (t.initializeInstanced if instanced else t.initializeBuffers)(sc, seed=5)
        t.initializeImageBuffers(width, height)
        t.set_counting(counting)
        c = None
        if cache:
            c = RadianceCache(t, seed=1)
            c.params = nrc_init_params(seed=3)
        t.run(TracerState(scene=sc, filmWidth=width, filmHeight=height, pixelStartOffset=first, pixelCount=count))
        return t.read_film().copy(), c.samples() if c else None


@pytest.mark.parametrize("width,height,first,count,spp,cache", [
    (613, 397, 0, 613 * 397, 1, False), (8, 60001, 0, 8 * 60001, 1, False), (7, 50003, 0, 7 * 50003, 1, False),
    (60007, 4, 0, 60007 * 4, 1, False), (100003, 3, 0, 100003 * 3, 1, False), (640, 400, 333, 190001, 1, False),
    (301, 203, 0, 301 * 203, 2, False), (613, 397, 0, 613 * 397, 1, True), (640, 401, 77, 201113, 1, True),
    (37, 29, 5, 1001, 1, False), (37, 29, 0, 1073, 1, True)])
def test_camera_rays_match_generated(width, height, first, count, spp, cache):
    sc = small_room(width=width, height=height)
    sc.settings.update(multi_sample_count_sqrt=spp, path_sample_count=1, max_path_length=4, russian_roulette_depth=0)
    film, samples = _render(sc, width, height, first, count, False, cache, False)
    ref, ref_samples = _render(sc, width, height, first, count, True, cache, False)
    assert np.array_equal(film, ref), f"{(film != ref).any(axis=1).sum()} pixels differ"
    if cache:
        assert samples.shape[0] > 0 and np.array_equal(samples, ref_samples)


@pytest.mark.parametrize("width,height,first,count", [(613, 397, 0, 613 * 397), (640, 400, 333, 190001)])
def test_two_level_camera_rays(width, height, first, count):
    sc = heightfield_blobs_instanced(instances=5, blob_level=2, hf_nx=40, hf_nz=20, dielectric_fraction=0.3)
    sc.width, sc.height = width, height
    sc.settings["max_path_length"] = 3
    film, _ = _render(sc, width, height, first, count, False, False, True)
    ref, _ = _render(sc, width, height, first, count, True, False, True)
    assert np.array_equal(film, ref), f"{(film != ref).any(axis=1).sum()} pixels differ"
