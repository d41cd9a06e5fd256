"""Two-level scenes of overlapping triangles in common planes: rounding puts
hits before the entries of the boxes around them, and where two triangles lie
that near the order of the walk decides which one is seen. Uncounted films
(4-wide trees for the bounces) see what the counted render (binary trees) sees,
bit for bit: sheets within a mesh, the walls of a room, and sheets that lie in
one plane as instances, translated, turned and scaled."""

from __future__ import annotations

import numpy as np
import pytest

from raycer_gb300 import scenes
from raycer_gb300.tracer import CudaTracer, TracerState

pytestmark = pytest.mark.gpu


def _sheet(rng, n, axis, at, reach, size):
    v = (rng.uniform(-reach, reach, size=(n, 1, 3)) + rng.normal(scale=size, size=(n, 3, 3))).reshape(n, 9)
    v[:, axis::3] = at
    return v.astype(np.float32).astype(np.float64)


def _scene(kind):
    rng = np.random.default_rng(8)
    turns = [dict()]
    if kind == "small triangles":
        v = _sheet(rng, 600, 2, -0.5, 1.0, 0.1)
    elif kind == "room":
        v = np.concatenate([_sheet(rng, 60, axis, s, 1.2, 0.5) for axis in range(3) for s in (-1.3, 1.3)])
    else:
        v = _sheet(rng, 200, 2, -0.5, 1.0, 0.4)
    if kind == "instances":
        turns += [dict(translate=(0.31, 0.17, 0.0)), dict(rotate=(0.0, 0.0, 90.0)), dict(rotate=(0.0, 0.0, 37.0)),
                  dict(rotate=(180.0, 0.0, 0.0), translate=(0.0, 0.0, -1.0)),
                  dict(scale=(0.7, 1.3, 1.0), translate=(-0.2, 0.1, 0.0))]
    ground = np.array([[-9.0, -2.0, -9.0, -9.0, -2.0, 9.0, 9.0, -2.0, 9.0],
                       [-9.0, -2.0, -9.0, 9.0, -2.0, 9.0, 9.0, -2.0, -9.0]])
    mats = [scenes.Material(diffuse=(0.1 + 0.2 * k, 0.9 - 0.2 * k, 0.5)) for k in range(4)]
    mats.append(scenes.Material(diffuse=(0.0, 0.0, 0.0), emittance=(3.0, 3.0, 3.0), is_emissive=True))
    insts = [scenes.InstanceDesc(mesh=0, **t) for t in turns] + [scenes.InstanceDesc(mesh=1)]
    camera = scenes.CameraDesc(position=(0.0, 0.0, 1.0) if kind == "room" else (0.2, 0.1, 3.0), fov=60.0)
    return scenes.InstancedScene(kind, [(v, (np.arange(len(v)) % 5).astype(np.uint32)), (ground, np.zeros(2, np.uint32))],
                                 insts, mats, camera, 64, 48,
                                 settings=dict(tracer="path", max_path_length=8, miss_radiance=(1.0, 1.0, 1.0)))


@pytest.mark.parametrize("width,height", [(64, 48), (500, 400)])
@pytest.mark.parametrize("kind", ["small triangles", "sheet", "room", "instances"])
def test_films(kind, width, height):
    sc = _scene(kind)
    films, rays = [], []
    for counting in (False, True):
        with CudaTracer(0) as t:
            t.initializeInstanced(sc, seed=5)
            t.initializeImageBuffers(width, height)
            t.set_counting(counting)
            t.run(TracerState(scene=sc, filmWidth=width, filmHeight=height, pixelCount=width * height))
            films.append(t.read_film().copy())
            rays.append(t.stats()["rays_traced"])
    assert rays[0] == rays[1]
    assert np.array_equal(films[0], films[1]), f"{(films[0] != films[1]).any(axis=1).sum()} pixels differ"
