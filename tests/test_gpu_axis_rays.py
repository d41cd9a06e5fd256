"""Rays with a direction component of zero whose origin lies in the plane of a
box: the box test's product is then 0 * inf, and in x the box is hit with a
NaN entry distance. Rays along the axes at the vertices of grids and boxes are
this case. Casts on both sides of the dispatch's lines equal the float32
oracle's bit for bit; films whose camera and bounce rays stay in such a plane
equal the counted render's, in one-level and two-level scenes."""

from __future__ import annotations

import ctypes as C
from itertools import product

import numpy as np
import pytest

import oracle
from raycer_gb300 import _native as N
from raycer_gb300 import scenes
from raycer_gb300.tracer import RAY_DTYPE, CudaTracer

from helpers import small_room
from test_gpu_cast import _edge_rays
from test_gpu_cast_tree import grow_tree

pytestmark = pytest.mark.gpu

ORDERS = [N.RC_ORDER_REFERENCE, N.RC_ORDER_NEAREST]
FAR = np.float32(3.0e38)


def _compare(sc, rays, order, any_hit=False):
    with CudaTracer(0) as t:
        t.initializeBuffers(sc)
        assert grow_tree(t) > 0
        hits = t.cast(rays, any_hit=any_hit, order=order)
    prim, tt, u, v, _ = oracle.Oracle(sc).cast32(rays, any_hit=any_hit, order=order)
    assert np.array_equal(hits["prim"], prim), int((hits["prim"] != prim).sum())
    for k, ref in (("t", tt), ("u", u), ("v", v)):
        assert np.array_equal(hits[k], ref, equal_nan=True)
    return prim


@pytest.mark.parametrize("n", [777, 32_768, 400_000, 1_300_000])
@pytest.mark.parametrize("direction", [(0.0, -1.0, 0.0), (-0.0, -1.0, -0.0), (0.0, 1.0, 0.0), (0.0, -1.0, 0.3)])
@pytest.mark.parametrize("order", ORDERS)
def test_rays_at_grid_vertices(n, direction, order):
    sc = scenes.heightfield_scene(nx=256, nz=128)
    at = np.unique(sc.vertices.reshape(-1, 3).astype(np.float32), axis=0)
    at = np.concatenate([at, (at[:-1] + at[1:]) * np.float32(0.5)])
    rays = np.zeros(n, RAY_DTYPE)
    rays["origin"] = np.resize(np.random.default_rng(1).permutation(at), (n, 3))
    rays["origin"][:, 1] = -10.0 * np.sign(direction[1])
    rays["direction"] = np.float32(direction)
    rays["t_max"] = FAR
    assert (_compare(sc, rays, order) >= 0).mean() > 0.6


def _cubes(leaf):
    """Cubes on a coarse grid: faces, edges and vertices coincide."""
    rng = np.random.default_rng(3)
    corner = np.array(list(product((0, 1), repeat=3)), np.float64)
    tris = []
    for _ in range(300):
        p = corner * rng.integers(1, 5) * 0.25 + rng.integers(-8, 8, 3) * 0.25
        for axis in range(3):
            for side in (0, 1):
                f = p[corner[:, axis] == side]
                tris += [f[[0, 1, 2]].ravel(), f[[1, 3, 2]].ravel()]
    v = np.array(tris)
    return scenes.SceneDesc("cubes", v, np.zeros(len(v), np.uint32), [scenes.Material(diffuse=(0.6, 0.6, 0.6))],
                            scenes.CameraDesc(position=(0.0, 0.0, 4.0), fov=50.0), 64, 48, max_leaf_size=leaf)


@pytest.mark.parametrize("n", [5_000, 100_000, 400_000, 1_300_000])
@pytest.mark.parametrize("leaf", [1, 4])
@pytest.mark.parametrize("order,any_hit", [(N.RC_ORDER_REFERENCE, False), (N.RC_ORDER_NEAREST, False),
                                           (N.RC_ORDER_NEAREST, True)])
def test_axis_rays_among_cubes(n, leaf, order, any_hit):
    rng = np.random.default_rng(n)
    rays = np.zeros(n, RAY_DTYPE)
    rays["origin"] = rng.integers(-16, 17, size=(n, 3)) * 0.125
    d = rng.integers(-1, 2, size=(n, 3)).astype(np.float32)
    d[(d == 0.0).all(axis=1)] = (0.0, 0.0, 1.0)
    rays["direction"] = np.where((d == 0.0) & (rng.random((n, 3)) < 0.5), np.float32(-0.0), d)
    rays["t_max"] = np.where(rng.random(n) < 0.5, FAR, np.float32(1.0))
    _compare(_cubes(leaf), rays, order, any_hit)


@pytest.mark.parametrize("order,any_hit", [(N.RC_ORDER_REFERENCE, False), (N.RC_ORDER_NEAREST, False),
                                           (N.RC_ORDER_NEAREST, True)])
def test_many_edge_rays(order, any_hit):
    rays = np.resize(_edge_rays(), 1_300_000)
    _compare(small_room(clutter=500), rays, order, any_hit)


def _terrain_under_glass():
    """A terrain whose grid has a column at x = 0, two glass panes above it."""
    hf = scenes.heightfield_scene(nx=65, nz=33)
    r = 30.0
    panes = np.concatenate([[[-r, y, -r, -r, y, r, r, y, r], [-r, y, -r, r, y, r, r, y, -r]] for y in (3.0, 3.5)])
    mats = [scenes.Material(diffuse=(0.8, 0.8, 0.8)), scenes.Material(dielectric=True, ior=1.5)]
    return scenes.InstancedScene("terrain under glass",
                                 [(hf.vertices, np.zeros(len(hf.vertices), np.uint32)), (panes, np.ones(4, np.uint32))],
                                 [scenes.InstanceDesc(mesh=0), scenes.InstanceDesc(mesh=1)], mats, hf.camera, 64, 48,
                                 settings=dict(tracer="path", max_path_length=6, miss_radiance=(1.0, 1.0, 1.0)))


def _plane_film(sc, two_level, width, height, counting):
    """The camera at x = 0 above the panes; every camera ray stays in that plane."""
    with CudaTracer(0) as t:
        if two_level:
            t.initializeInstanced(sc, seed=5)
        else:
            t.initializeBuffers(sc.flatten(), seed=5)
        t.initializeImageBuffers(width, height)
        t.set_counting(counting)
        cam = N.rc_camera()
        cam.position[:] = (0.0, 6.0, 0.0)
        cam.forward[:] = (0.0, -1.0, 0.0)
        cam.right[:] = (0.0, 0.0, 1.2)
        cam.up[:] = (0.0, 0.0, 0.3)
        cam.image_plane_center[:] = (0.0, 5.0, 0.0)
        cam.image_plane_width, cam.image_plane_height = width - 1.0, height - 1.0
        cam.aspect_ratio = height / width
        t.set_camera(cam)
        t._check(t._lib.rc_render(t.handle, 0, width * height, None, C.byref(C.c_uint64(0))), "render")
        return t.read_film().copy(), t.stats()["rays_traced"]


@pytest.mark.parametrize("two_level,width,height", [(True, 64, 48), (True, 400, 400), (False, 64, 48), (False, 400, 400)])
def test_films_in_a_box_plane(two_level, width, height):
    sc = _terrain_under_glass()
    film, rays = _plane_film(sc, two_level, width, height, False)
    ref, ref_rays = _plane_film(sc, two_level, width, height, True)
    assert rays == ref_rays
    assert np.array_equal(film, ref), f"{(film != ref).any(axis=1).sum()} pixels differ"
    # most paths go through the panes, down to the terrain and on
    assert rays > 3.5 * width * height
