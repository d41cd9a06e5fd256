"""The work that performance of this framework is measured on.

Each case is one call (or the calls of one frame) of the public entry points,
at sizes of the benchmark, the tests and the scene descriptions in
``raycer_gb300/scenes.py``: RAY frames, batches of ray queries from the host
and on the device, caller-ray frames, path-traced frames of plain, cached and
two-level scenes, and several scenes in one launch.

The scene of a case is fixed by the case; the seed sets what changes between
two frames or calls of a program: the camera, the light, the rays, the random
stream. A frame ends with its result where a program wants it: the records or
the tone-mapped image in the program's own page-locked buffer, or device
memory for device batches.
"""

from __future__ import annotations

import ctypes as C
import math
import random
from functools import lru_cache

import numpy as np
import torch

from raycer_gb300 import _native as N
from raycer_gb300 import scenes
from raycer_gb300.batch import Batch
from raycer_gb300.nrc import RadianceCache
from raycer_gb300.tracer import HIT_DTYPE, RAY_DTYPE, CudaTracer, TracerState

FAR = 3.0e38


def listed() -> list[dict]:
    return [
        # A thumbnail of a small scene: what a RAY call costs by itself.
        dict(name="ray_preview", kind="ray", nx=96, nz=48, width=160, height=90, order=1, first=0, part=1.0),
        # The benchmark's headline frame: primary + shadow rays, 1M triangles.
        dict(name="ray_1080p", kind="ray", nx=1024, nz=512, width=1920, height=1080, order=1, first=0, part=1.0),
        # A pixel range of an odd-sized film in the reference's traversal
        # order: a network worker's share of a frame, checked against the CPU.
        dict(name="ray_range", kind="ray", nx=300, nz=151, width=1237, height=701, order=0, first=301, part=0.37),
        # A few hundred picking / visibility queries from host arrays.
        dict(name="cast_pick", kind="cast", nx=1024, nz=512, rays=777, any_hit=0, where="host"),
        # Millions of incoherent closest-hit queries on device buffers.
        dict(name="cast_4m", kind="cast", nx=1024, nz=512, rays=4_000_000, any_hit=0, where="device"),
        # The caller's own primary rays of a 1080p frame, host to host.
        dict(name="frame_host", kind="frame", nx=1024, nz=512, width=1920, height=1080),
        # A one-sample preview of a small room: launches and latency of PATH.
        dict(name="path_preview", kind="room", clutter=300, extra=0, width=64, height=48, spp_sqrt=1, depth=4, rr=0,
             filter="box"),
        # The room of the reference's own configuration, 16 CMJ samples.
        dict(name="path_room", kind="room", clutter=2000, extra=0, width=320, height=240, spp_sqrt=4, depth=4, rr=0,
             filter="box"),
        # The path-tracing headline: 1M triangles, 1080p, four segments.
        dict(name="path_1m", kind="terrain", nx=1024, nz=512, width=1920, height=1080, depth=4),
        # A radiance-cache frame of the closed 5M-triangle scene, 12 segments.
        dict(name="cache_box", kind="blobs", cache=1, enclosed=1, instances=200, level=5, nx=1024, nz=512, width=1920,
             height=1080, depth=12),
        # Instanced blobs, a third of them glass, under a sky: two-level BVH.
        dict(name="path_instanced", kind="instanced", instances=200, level=5, nx=1024, nz=512, glass=0.3, width=1920,
             height=1080, depth=12),
        # Rooms of uneven size, resolution and sample count as one launch.
        dict(name="batch_rooms", kind="batch", scenes=6, n_min=1000, n_max=300_000, res_min=256, res_max=768,
             depth=8, rr=3),
    ]


def _log(rng: random.Random, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["ray", "ray", "cast", "cast", "frame", "room", "room", "terrain", "blobs", "instanced", "batch"])
    nx, nz = _log(rng, 96, 1024), _log(rng, 48, 512)
    width, height = _log(rng, 160, 1920), _log(rng, 90, 1080)
    if kind == "ray":
        part = rng.choice([1.0, 1.0, round(rng.uniform(0.1, 0.9), 3)])
        return dict(kind=kind, nx=nx, nz=nz, width=width, height=height, order=rng.choice([1, 1, 0]),
                    first=0 if part == 1.0 else rng.randrange(0, width * height // 20), part=part)
    if kind == "cast":
        return dict(kind=kind, nx=nx, nz=nz, rays=_log(rng, 500, 4_000_000), any_hit=rng.choice([0, 0, 1]),
                    where=rng.choice(["host", "device"]))
    if kind == "frame":
        return dict(kind=kind, nx=nx, nz=nz, width=width, height=height)
    if kind == "room":
        spp_sqrt = rng.randint(1, 4)
        return dict(kind=kind, clutter=_log(rng, 200, 2000), extra=rng.choice([0, _log(rng, 1000, 200_000)]),
                    width=_log(rng, 64, 320), height=_log(rng, 48, 240), spp_sqrt=spp_sqrt, depth=rng.randint(2, 8),
                    rr=rng.choice([0, 3]), filter=rng.choice(["box", "box", "mitchell", "gaussian"]))
    if kind == "terrain":
        return dict(kind=kind, nx=nx, nz=nz, width=width, height=height, depth=rng.randint(2, 8))
    if kind == "blobs":
        return dict(kind=kind, cache=rng.choice([0, 1]), enclosed=rng.choice([0, 1]), instances=rng.randint(3, 80),
                    level=rng.randint(2, 4), nx=nx, nz=nz, width=width, height=height, depth=rng.randint(4, 12))
    if kind == "instanced":
        return dict(kind=kind, instances=rng.randint(3, 200), level=rng.randint(2, 5), nx=nx, nz=nz,
                    glass=round(rng.uniform(0.0, 0.5), 2), width=width, height=height, depth=rng.randint(3, 12))
    return dict(kind=kind, scenes=rng.randint(2, 6), n_min=1000, n_max=_log(rng, 2000, 100_000), res_min=128,
                res_max=rng.randint(160, 512), depth=rng.randint(3, 8), rr=rng.choice([0, 3]))


# ---------------------------------------------------------------------------
# Scenes (geometry only; the camera and settings of a state are its own copy).


@lru_cache(maxsize=4)
def _terrain(nx: int, nz: int):
    return scenes.heightfield_scene(nx=nx, nz=nz)


@lru_cache(maxsize=4)
def _geometry(kind: str, key: tuple):
    c = dict(key)
    if kind == "terrain":
        return scenes.heightfield_path_scene(nx=c["nx"], nz=c["nz"])
    if kind == "room":
        return scenes.room_with_extra(1, c["extra"], 320, 240, 1) if c["extra"] else scenes.room_scene(1, c["clutter"])
    if kind == "blobs":
        return scenes.heightfield_blobs_scene(instances=c["instances"], blob_level=c["level"], hf_nx=c["nx"],
                                              hf_nz=c["nz"], enclosed=bool(c["enclosed"]))
    return scenes.heightfield_blobs_instanced(instances=c["instances"], blob_level=c["level"], hf_nx=c["nx"],
                                              hf_nz=c["nz"], dielectric_fraction=c["glass"])


def _scene(case: dict):
    """A copy of the case's scene record (the geometry arrays are shared)."""
    import copy

    if case["kind"] in ("ray", "cast", "frame"):
        sc = _terrain(case["nx"], case["nz"])
    else:
        keys = ("nx", "nz", "clutter", "extra", "instances", "level", "enclosed", "glass")
        sc = _geometry(case["kind"], tuple((k, case[k]) for k in keys if k in case))
    sc = copy.copy(sc)
    sc.camera = copy.copy(sc.camera)
    sc.settings = dict(sc.settings)
    if "width" in case:
        sc.width, sc.height = case["width"], case["height"]
    return sc


def _aim(sc, rng: random.Random) -> None:
    """Another viewpoint of the same scene."""
    x, y, z = sc.camera.position
    room = sc.name.startswith("room")
    r = 0.15 if room else 1.5
    sc.camera.position = (x + rng.uniform(-r, r), y + rng.uniform(-0.3, 0.3) * r, z + rng.uniform(-0.3, 0.0) * r)
    sc.camera.yaw = rng.uniform(-3.0, 3.0)
    sc.camera.pitch = sc.camera.pitch + rng.uniform(-2.0, 2.0)


def _sunlight(rng: random.Random) -> tuple:
    """Travel direction of a light 25 to 80 degrees above the horizon."""
    el, az = math.radians(rng.uniform(25.0, 80.0)), rng.uniform(0.0, 2.0 * math.pi)
    return (-math.cos(el) * math.cos(az), -math.sin(el), -math.cos(el) * math.sin(az))


def _rays(case: dict, seed: int) -> np.ndarray:
    """Queries over the terrain: origins in its air space, uniform directions;
    half of them with a far limit, as visibility and ambient-occlusion rays have."""
    g = np.random.default_rng(seed)
    n = case["rays"]
    rays = np.zeros(n, RAY_DTYPE)
    rays["origin"] = g.random((n, 3), np.float32) * np.float32([18.0, 3.0, 9.0]) + np.float32([-9.0, 0.8, -4.5])
    d = g.standard_normal((n, 3), np.float32)
    rays["direction"] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays["t_max"] = np.where(g.random(n, np.float32) < 0.5, np.float32(FAR), 0.5 + 4.0 * g.random(n, np.float32))
    return rays


def _view(sc):
    """Camera position and the frame of the image plane in 64 bits: the
    reference's perspective camera (forward from pitch and yaw, right and up
    about ALMOST_UP, plane distance 0.5 / tan(fov / 2), horizontal fov)."""
    p, y = math.radians(sc.camera.pitch), math.radians(sc.camera.yaw)
    unit = lambda v: v / np.linalg.norm(v)  # noqa: E731
    fwd = unit(np.array([-math.sin(y) * math.cos(p), math.sin(p), -math.cos(y) * math.cos(p)]))
    right = unit(np.cross(fwd, [0.0001, 1.0, 0.0001]))
    up = unit(np.cross(right, fwd))
    pos = np.array(sc.camera.position, np.float64)
    return pos, pos + fwd * (0.5 / math.tan(math.radians(sc.camera.fov) / 2.0)), right, up


def _camera_rays(sc) -> tuple[np.ndarray, np.ndarray]:
    """Origin and unit directions of every pixel's ray, in 64 bits."""
    pos, centre, right, up = _view(sc)
    px, py = np.meshgrid(np.arange(sc.width, dtype=np.float64), np.arange(sc.height, dtype=np.float64))
    dx = px.ravel() / (sc.width - 1) - 0.5
    dy = (py.ravel() / (sc.height - 1) - 0.5) * (sc.height / sc.width)
    d = centre - pos + dx[:, None] * right + dy[:, None] * up
    return pos, d / np.linalg.norm(d, axis=1, keepdims=True)


# ---------------------------------------------------------------------------


class State:
    """What a program holds between two frames."""

    def close(self):
        for h in (getattr(self, "tracer", None), getattr(self, "batch", None)):
            if h is not None:
                h.close()

    def __del__(self):
        self.close()


def _pinned(n: int, dtype) -> torch.Tensor:
    t = torch.empty((n, 4), dtype=dtype, pin_memory=True)
    t.zero_()
    return t


def _ptr(t: torch.Tensor) -> C.c_void_p:
    return C.c_void_p(t.data_ptr())


def _settings(case: dict, sc) -> None:
    if case["kind"] == "room":
        sc.settings.update(multi_sample_count_sqrt=case["spp_sqrt"], max_path_length=case["depth"],
                           russian_roulette_depth=case["rr"], filter=case["filter"])
    elif case["kind"] in ("terrain", "blobs", "instanced"):
        sc.settings["max_path_length"] = case["depth"]


def _batch_scenes(case: dict, rng: random.Random) -> list:
    """Rooms whose extra triangles, film sizes and sample counts cover the case's ranges."""
    out = []
    k = case["scenes"]
    for i in range(k):
        f = i / max(1, k - 1)
        extra = int(round(math.exp(math.log(case["n_min"]) + f * (math.log(case["n_max"]) - math.log(case["n_min"])))))
        res = int(round(case["res_min"] + ((i * 2) % k) / max(1, k - 1) * (case["res_max"] - case["res_min"])))
        sc = scenes.room_with_extra(3000 + i, extra, res, res, 1 + (i * 5) % 3, max_path_length=case["depth"],
                                    rr_depth=case["rr"])
        _aim(sc, rng)
        out.append(sc)
    return out


def prepare(case: dict, seed: int) -> State:
    rng = random.Random(seed)
    s = State()
    s.kind = case["kind"]
    s.cache = None
    if s.kind == "batch":
        s.batch = Batch(0)
        s.images = []
        for sc in _batch_scenes(case, rng):
            s.batch.add_scene(sc, seed=rng.randrange(1 << 30))
            s.images.append(_pinned(sc.width * sc.height, torch.float32))
        return s
    sc = _scene(case)
    _settings(case, sc)
    s.tracer = t = CudaTracer(0)
    if s.kind == "cast":
        t.initializeBuffers(sc)
        rays = _rays(case, seed)
        s.any_hit = bool(case["any_hit"])
        s.device = case["where"] == "device"
        if s.device:
            s.rays = torch.from_numpy(rays.view(np.float32).reshape(-1, 8)).cuda()
            s.hits = torch.zeros((rays.shape[0], 4), dtype=torch.int32, device="cuda")
        else:
            s.rays = rays
        return s
    _aim(sc, rng)
    if s.kind in ("ray", "frame"):
        sc.light_direction = _sunlight(rng)
    if s.kind == "instanced":
        t.initializeInstanced(sc, seed=rng.randrange(1 << 30))
    else:
        t.initializeBuffers(sc, seed=rng.randrange(1 << 30))
    t.initializeImageBuffers(sc.width, sc.height)
    n = sc.width * sc.height
    if s.kind == "frame":
        pos, d = _camera_rays(sc)
        rays = torch.empty((n, 8), dtype=torch.float32, pin_memory=True)
        rays[:, 0:3] = torch.from_numpy(pos)
        rays[:, 3] = 0.0
        rays[:, 4:7] = torch.from_numpy(d)
        rays[:, 7] = FAR
        s.rays, s.out = rays, _pinned(n, torch.int32)
        return s
    if s.kind == "ray":
        t.set_traversal_order(case["order"])
        count = n if case["part"] == 1.0 else max(1, int(n * case["part"]))
        s.out = _pinned(n, torch.int32)
        s.state = TracerState(scene=sc, filmWidth=sc.width, filmHeight=sc.height, pixelStartOffset=case["first"],
                              pixelCount=count)
        return s
    s.image = _pinned(n, torch.float32)
    s.state = TracerState(scene=sc, filmWidth=sc.width, filmHeight=sc.height, pixelCount=n)
    if case.get("cache"):
        # every frame starts from the same saved weights, as the first frame after a cut does
        s.cache = RadianceCache(t, seed=1)
        s.weights = s.cache.params
    return s


def _records(rec: torch.Tensor) -> dict:
    return {"prim": rec[:, 0], "t": rec.view(torch.float32)[:, 1], "occluder": rec[:, 2], "flags": rec[:, 3]}


def _hits(rec: torch.Tensor) -> dict:
    f = rec.view(torch.float32)
    return {"prim": rec[:, 0], "t": f[:, 1], "u": f[:, 2], "v": f[:, 3]}


def run(s: State):
    if s.kind == "batch":
        s.batch.render()
        for i, img in enumerate(s.images):
            s.batch._check(s.batch._lib.rc_batch_resolve(s.batch._h, i, None, _ptr(img)), "resolve")
        return s.images
    t = s.tracer
    if s.kind == "cast":
        if s.device:
            t._check(t._lib.rc_cast_device(t.handle, _ptr(s.rays), s.rays.shape[0], int(s.any_hit),
                                           N.RC_ORDER_NEAREST, _ptr(s.hits)), "cast")
            return _hits(s.hits)
        hits = t.cast(s.rays, any_hit=s.any_hit)
        return {k: hits[k] for k in HIT_DTYPE.names}
    if s.kind == "frame":
        t._check(t._lib.rc_cast_with_shadow(t.handle, _ptr(s.rays), s.rays.shape[0], N.RC_ORDER_NEAREST, _ptr(s.out)),
                 "cast_with_shadow")
        return _records(s.out)
    if s.cache is not None:
        s.cache.params = s.weights
    t.run(s.state)
    if s.kind == "ray":
        t._check(t._lib.rc_read_cast(t.handle, _ptr(s.out)), "read_cast")
        return _records(s.out)
    t._check(t._lib.rc_resolve(t.handle, _ptr(s.image)), "resolve")
    return s.image


# ---------------------------------------------------------------------------


def _closest(tri: np.ndarray, origin: np.ndarray, d: np.ndarray, limit: np.ndarray) -> tuple:
    """Closest hits of rays with every triangle (Moeller-Trumbore), in 64 bits:
    distance, u, v; a miss is -1, 0, 0."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    v = torch.from_numpy(np.ascontiguousarray(tri, np.float64)).to(dev)
    v0, e1, e2 = v[:, 0:3], v[:, 3:6] - v[:, 0:3], v[:, 6:9] - v[:, 0:3]
    # every triple product of the test as a dot product with a vector of the triangle or of the ray
    n = torch.linalg.cross(e1, e2)
    m1, m2, n0 = torch.linalg.cross(e1, v0), torch.linalg.cross(v0, e2), (n * v0).sum(1)
    out = [[], [], []]
    step = max(1, (1 << 27) // max(1, v.shape[0]))
    for a in range(0, d.shape[0], step):
        D = torch.from_numpy(d[a:a + step]).to(dev)
        O = torch.from_numpy(np.broadcast_to(origin, d.shape)[a:a + step].copy()).to(dev)
        far = torch.from_numpy(limit[a:a + step]).to(dev)
        M = torch.linalg.cross(O, D)  # moment of the ray
        det = -(D @ n.T)
        u = (M @ e2.T + D @ m2.T) / det
        w = (D @ m1.T - M @ e1.T) / det
        t = (O @ n.T - n0) / det
        ok = (det.abs() >= 1.1920928955078125e-7) & (u >= 0) & (u <= 1) & (w >= 0) & (u + w <= 1) & (t >= 0)
        t = torch.where(ok & (t <= far[:, None]), t, math.inf)
        best, at = t.min(1)
        hit = torch.isfinite(best)
        out[0].append(torch.where(hit, best, -1.0).cpu())
        out[1].append(torch.where(hit, u.gather(1, at[:, None])[:, 0], 0.0).cpu())
        out[2].append(torch.where(hit, w.gather(1, at[:, None])[:, 0], 0.0).cpu())
    return tuple(torch.cat(o) for o in out)


def exact(case: dict, seed: int):
    """Distances (and barycentrics) of the small ray batches in 64 bits, over
    all triangles. None for the large ones, where that takes minutes, and for
    path-traced images: a pixel's value hangs on the last bit of every bounce."""
    if case["kind"] == "cast" and case["any_hit"] == 0 and case["rays"] * case["nx"] * case["nz"] <= 4e9:
        sc = _scene(case)
        r = _rays(case, seed)
        t, u, v = _closest(sc.vertices, r["origin"].astype(np.float64), r["direction"].astype(np.float64),
                           r["t_max"].astype(np.float64))
        return {"prim": None, "t": t, "u": u, "v": v}
    if case["kind"] == "ray" and case["part"] == 1.0 and case["width"] * case["height"] * case["nx"] * case["nz"] <= 4e9:
        sc = _scene(case)
        _aim(sc, random.Random(seed))
        pos, d = _camera_rays(sc)
        t, _, _ = _closest(sc.vertices, pos, d, np.full(d.shape[0], np.inf))
        return {"prim": None, "t": t, "occluder": None, "flags": None}
    return None


def work(case: dict) -> dict:
    """Bytes: the scene arrays a frame can touch (36 B of vertices per
    triangle, at most one leaf of four per ray), the rays and the results,
    each once. Floating-point operations: one descent of a balanced tree per
    ray (two 18-operation box tests per level) and one triangle test (45)."""
    kind = case["kind"]
    px = case.get("width", 0) * case.get("height", 0)
    terrain = 2 * (case.get("nx", 2) - 1) * (case.get("nz", 2) - 1)
    io, segments = 16 * px, 1.0
    if kind == "ray":
        rays = 2 * px * case["part"]
        io, tris = 16 * px, terrain
    elif kind == "cast":
        rays, tris = case["rays"], terrain
        io = 48 * rays
    elif kind == "frame":
        rays, tris = 2 * px, terrain
        io = 48 * px
    elif kind == "room":
        tris = 12 + (2000 + case["extra"] if case["extra"] else case["clutter"])
        rays = px * case["spp_sqrt"] ** 2
        segments = min(case["depth"], 3)
    elif kind == "terrain":
        rays, tris, segments = px, terrain + 2, 1.8
    elif kind in ("blobs", "instanced"):
        rays = px
        tris = terrain + case["instances"] * 20 * 4 ** case["level"]
        segments = 3.0
    else:
        rays = io = tris = 0
        for i in range(case["scenes"]):
            k = case["scenes"]
            res = case["res_min"] + ((i * 2) % k) / max(1, k - 1) * (case["res_max"] - case["res_min"])
            rays += res * res * (1 + (i * 5) % 3) ** 2
            io += 16 * res * res
            tris += 2012 + case["n_min"] * (case["n_max"] / case["n_min"]) ** (i / max(1, k - 1))
        segments = 3.0
    per_ray = 36.0 * math.log2(max(2.0, tris / 4.0)) + 45.0
    return {"bytes": float(io + min(36.0 * tris, 4 * 36.0 * rays)), "flops": float(rays * segments * per_ray)}
