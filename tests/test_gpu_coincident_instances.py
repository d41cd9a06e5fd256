"""Instances of one mesh at one place, of different materials: the closest hit
is the same triangle at the same distance in each, and the walk's order decides
whose material is seen. Uncounted films (4-wide trees for the bounces) see what
the counted render (binary trees) sees, bit for bit."""

from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from raycer_gb300 import scenes
from raycer_gb300.tracer import CudaTracer, TracerState

pytestmark = pytest.mark.gpu


def _scene(blobs, copies):
    sc = scenes.heightfield_blobs_instanced(instances=blobs, blob_level=2, hf_nx=64, hf_nz=32, width=640, height=360)
    first = len(sc.materials)
    sc.materials = list(sc.materials) + [
        scenes.Material(diffuse=(0.9, 0.1 + 0.8 * k / copies, 0.9 - 0.8 * k / copies)) for k in range(copies)]
    again = [dataclasses.replace(inst, material=first + k) for k in range(copies) for inst in sc.instances[1:]]
    rng = np.random.default_rng(blobs)
    sc.instances = list(sc.instances[:1]) + [(list(sc.instances[1:]) + again)[i]
                                             for i in rng.permutation(len(sc.instances) - 1 + len(again))]
    sc.settings.update(max_path_length=8, miss_radiance=(1.0, 1.0, 1.0))
    return sc


@pytest.mark.parametrize("blobs,copies", [(24, 3), (60, 15), (150, 3), (150, 7), (300, 1)])
def test_coincident_instances(blobs, copies):
    sc = _scene(blobs, copies)
    films, rays = [], []
    for counting in (False, True):
        with CudaTracer(0) as t:
            t.initializeInstanced(sc, seed=13)
            t.initializeImageBuffers(sc.width, sc.height)
            t.set_counting(counting)
            t.run(TracerState(scene=sc, filmWidth=sc.width, filmHeight=sc.height, pixelCount=sc.width * sc.height))
            films.append(t.read_film().copy())
            rays.append(t.stats()["rays_traced"])
    assert rays[0] == rays[1]
    assert np.array_equal(films[0], films[1]), f"{(films[0] != films[1]).any(axis=1).sum()} pixels differ"
