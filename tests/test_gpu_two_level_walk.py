"""Two-level scenes: the bounce kernel's walk over both levels (4-wide trees)
gives the films of the counted render, whose extend kernel nests the mesh walk
in the walk over the instances, bit for bit: one instance (the top-level root
is a leaf), two (one leaf of two), many overlapping ones, meshes of a single
leaf, glass, Russian roulette, one and two segments, radiance-cache lookups."""

from __future__ import annotations

import numpy as np
import pytest

from raycer_gb300 import scenes
from raycer_gb300.nrc import RadianceCache
from raycer_gb300.tracer import CudaTracer, TracerState

pytestmark = pytest.mark.gpu


def _scene(kind):
    if kind == "single leaf meshes":
        tri = np.array([[-2.0, -1.0, 0.0, 2.0, -1.0, 0.0, 0.0, 2.0, 0.0]])
        quad = np.array([[-4.0, -2.0, -4.0, -4.0, -2.0, 4.0, 4.0, -2.0, 4.0], [-4.0, -2.0, -4.0, 4.0, -2.0, 4.0, 4.0, -2.0, -4.0]])
        meshes = [(tri, np.zeros(1, np.uint32)), (quad, np.zeros(2, np.uint32))]
        insts = [scenes.InstanceDesc(mesh=1)] + [
            scenes.InstanceDesc(mesh=0, material=k % 3, scale=(0.5 + 0.1 * k,) * 3, rotate=(20.0 * k, 35.0 * k, 10.0 * k),
                                translate=(0.6 * (k - 4), 0.2 * k, -0.5 * k)) for k in range(9)]
        mats = [scenes.Material(diffuse=(0.7, 0.7, 0.7)), scenes.Material(diffuse=(0.8, 0.3, 0.2)),
                scenes.Material(dielectric=True, ior=1.5)]
        return scenes.InstancedScene(kind, meshes, insts, mats, scenes.CameraDesc(position=(0.0, 0.0, 8.0), fov=50.0), 64,
                                     36, settings=dict(tracer="path", max_path_length=6, miss_radiance=(1.0, 1.0, 1.0)))
    n = {"one instance": 0, "two instances": 1, "many": 40}[kind]
    return scenes.heightfield_blobs_instanced(instances=n, blob_level=2, hf_nx=64, hf_nz=32, width=64, height=36,
                                              dielectric_fraction=0.4)


def _film(sc, counting, cache):
    with CudaTracer(0) as t:
        t.initializeInstanced(sc, seed=13)
        t.initializeImageBuffers(sc.width, sc.height)
        if cache:
            RadianceCache(t)
        t.set_counting(counting)
        t.run(TracerState(scene=sc, filmWidth=sc.width, filmHeight=sc.height, pixelCount=sc.width * sc.height))
        return t.read_film().copy(), t.stats()["rays_traced"]


@pytest.mark.parametrize("depth,rr,cache", [(1, 0, False), (2, 0, False), (9, 3, False), (9, 0, True)])
@pytest.mark.parametrize("kind", ["one instance", "two instances", "many", "single leaf meshes"])
def test_films(kind, depth, rr, cache):
    sc = _scene(kind)
    sc.settings.update(max_path_length=depth, russian_roulette_depth=rr)
    film, rays = _film(sc, False, cache)
    ref, ref_rays = _film(sc, True, cache)
    assert np.array_equal(film, ref), f"{(film != ref).any(axis=1).sum()} pixels differ"
    assert rays == ref_rays
    assert film[:, :3].max() > 0.0
