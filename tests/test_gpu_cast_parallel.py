"""Large closest-hit casts of parallel and nearly parallel rays onto
overlapping triangles of one axis-aligned plane. Box rounding then decides
between equal hits for most rays (up to 99 % here), the casts list those to be
walked again alone, and whole warps of them finish together: the lists fill
faster than with random rays. The hits equal the float32 oracle's."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from raycer_gb300 import _native as N
from raycer_gb300 import scenes
from raycer_gb300.tracer import RAY_DTYPE, CudaTracer

from test_gpu_cast_tree import grow_tree

pytestmark = pytest.mark.gpu


def _sheet():
    rng = np.random.default_rng(8)
    n = 200
    v = (rng.uniform(-1.0, 1.0, size=(n, 1, 3)) + rng.normal(scale=0.4, size=(n, 3, 3))).reshape(n, 9)
    v[:, 2::3] = -0.5
    v = v.astype(np.float32).astype(np.float64)
    return scenes.SceneDesc("sheet", v, np.zeros(n, np.uint32), [scenes.Material(diffuse=(0.6, 0.6, 0.6))],
                            scenes.CameraDesc(position=(0.0, 0.0, 4.0), fov=50.0), 64, 48, max_leaf_size=4)


@pytest.mark.parametrize("height,spread", [(0.5, 0.0), (0.7, 1e-3), (1.3, 0.0), (1.3, 1e-3)])
def test_parallel_rays_onto_a_sheet(height, spread):
    sc = _sheet()
    rng = np.random.default_rng(17)
    n = 1_300_000
    rays = np.zeros(n, RAY_DTYPE)
    d = np.array((0.05, 0.02, -1.0)) + spread * rng.normal(size=(n, 3))
    rays["direction"] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays["origin"][:, :2] = rng.uniform(-0.7, 0.7, size=(n, 2))
    rays["origin"][:, 2] = height
    rays["t_max"] = 3.0e38
    with CudaTracer(0) as t:
        t.initializeBuffers(sc)
        assert grow_tree(t) > 0
        hits = t.cast(rays, order=N.RC_ORDER_NEAREST)
    prim, tt, u, v, _ = oracle.Oracle(sc).cast32(rays, any_hit=False, order=1)
    assert (prim >= 0).all()
    assert np.array_equal(hits["prim"], prim), int((hits["prim"] != prim).sum())
    for k, ref in (("t", tt), ("u", u), ("v", v)):
        assert np.array_equal(hits[k], ref)
