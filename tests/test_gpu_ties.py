"""Primitives at one distance, on a B200: which of them a ray meets.

Where two quads lie in a plane, faces of neighbouring boxes meet, or a sphere is in the scene twice, every ray there has
several closest hits, and the one it gets follows from the order in which the tree is walked: for closest-hit queries
and for the FP64 integrator the two-wide tree's. The persistent kernel walks that tree, so its image of lamps with a
color each, one pass of one segment, says which primitive each of its camera rays meets.
"""
import ctypes as C
from pathlib import Path

import numpy as np
import pytest

from raytracing_b200 import _abi

pytestmark = pytest.mark.gpu

GOLDEN = Path(__file__).resolve().parent / "golden"


def _v(x, y, z):
    return _abi.Vec3(float(x), float(y), float(z))


def _quad(q, u, v):
    return _abi.QuadDesc(q=_v(*q), u=_v(*u), v=_v(*v))


def _sphere(c, r):
    return _abi.SphereDesc(center=_v(*c), radius=r, uv_cos=1.0)


def _tilings(turn=0.0):
    # two tilings of one plane, the second half a tile off
    x, y = np.array([np.cos(turn), 0.3 * np.sin(turn), np.sin(turn)]), np.array([-0.2 * np.sin(turn), np.cos(turn), 0.1 * turn])
    return [_quad((i + s) * x + (j + s / 2) * y, x, y) for s in (0, 0.5) for i in range(-8, 8) for j in range(-8, 8)]


def _triangles():
    # the same of triangles, a mesh of its own each
    out = []
    for s in (0, 0.5):
        for i in range(-8, 8):
            for j in range(-8, 8):
                p = [(i + s, j + s / 2, 0), (i + s + 1, j + s / 2, 0), (i + s + 1, j + s / 2 + 1, 0), (i + s, j + s / 2 + 1, 0)]
                out += [[p[0], p[1], p[2]], [p[0], p[2], p[3]]]
    return out


def _twins():
    r = np.random.default_rng(3)
    one = [(r.uniform([-5, -4, -8], [5, 4, 0]), r.uniform(0.3, 1.0)) for _ in range(60)]
    return [_sphere(c, s) for c, s in one + one[::-1]]


SCENES = {"tilings": _tilings, "tilted": lambda: _tilings(0.7), "triangles": _triangles, "twins": _twins}


def _scene(rt, name, kind, depth):
    """The scene's shapes, each with a material of its own: a lamp whose color is its number, or a matte color."""
    shapes = SCENES[name]()
    n = len(shapes)
    textures, materials = (_abi.TextureDesc * n)(), (_abi.MaterialDesc * n)()
    lamps = kind == _abi.RT_DIFFUSE_LIGHT
    for k in range(n):
        textures[k] = _abi.TextureDesc(kind=_abi.RT_TEXTURE_SOLID)
        textures[k].rgb = _v(k + 1, 0, 0) if lamps else _v(k % 3 == 0, (k % 5) / 5, (k % 7) / 7)
        materials[k] = _abi.MaterialDesc(kind=kind, texture=k)
    cam = _abi.CameraDesc(image_width=160, image_height=120, sqrt_spp=1, max_depth=depth, center=_v(0, 0, 10),
                          sampling=_abi.RT_SAMPLING_MATERIAL)
    cam.pixel_delta_u, cam.pixel_delta_v = _v(1 / 160, 0, 0), _v(0, -1 / 160, 0)
    cam.pixel00_loc = _v(-0.5, 0.375, 9)
    if not lamps:
        cam.sky_bottom, cam.sky_top = _v(1, 1, 1), _v(0.5, 0.7, 1)
    desc = _abi.SceneDesc(materials=materials, material_count=n, textures=textures, texture_count=n, camera=cam)
    if name == "triangles":
        meshes, keep = (_abi.MeshDesc * n)(), []
        for k, corners in enumerate(shapes):
            keep.append(((C.c_float * 9)(*np.ravel(corners)), (C.c_uint32 * 3)(0, 1, 2)))
            meshes[k] = _abi.MeshDesc(positions=keep[-1][0], vertex_count=3, indices=keep[-1][1], triangle_count=1, material=k)
        desc.meshes, desc.mesh_count = meshes, n
    else:
        for k, shape in enumerate(shapes):
            shape.material = k
        array = (type(shapes[0]) * n)(*shapes)
        if name == "twins":
            desc.spheres, desc.sphere_count = array, n
        else:
            desc.quads, desc.quad_count = array, n
    return rt.Scene(C.pointer(desc))


@pytest.mark.parametrize("name", SCENES)
def test_a_querys_hit_among_the_nearest(rt, name):
    scene = _scene(rt, name, _abi.RT_DIFFUSE_LIGHT, 1)
    assert scene.stats()["flat"] == 0
    session = rt.Session(scene, seed=7, form="persistent")
    session.render_to(1)
    want = session.pixels()[..., 0].ravel().astype(np.int64) - 1
    o, d = scene.camera_rays(7, 0)
    ids, ts = scene.closest_hits(o, d)
    met = want >= 0
    assert met.mean() > 0.05
    assert np.array_equal(ids[met], want[met])
    assert (ids >= 0).sum() >= met.sum() and np.isfinite(ts[met]).all()


def _fp64_ids(rt, name):
    session = rt.Session(_scene(rt, name, _abi.RT_DIFFUSE_LIGHT, 1), seed=7, arithmetic="float64")
    session.render_to(1)
    return session.pixels()[..., 0].astype(np.int64) - 1


@pytest.mark.parametrize("name", [n for n in SCENES if n != "triangles"])
def test_fp64_paths_hits_among_the_nearest(rt, name):
    # as rendered by a lane's walk of the two-wide tree in double, path by path, which a path that meets a tie still takes
    want = np.load(GOLDEN / "fp64_ties.npz")[name]
    assert (want >= 0).mean() > 0.05
    assert np.array_equal(_fp64_ids(rt, name), want)


def test_fp64_ties_in_many_launches(rt):
    # paths dropped at a tie and rendered again, in one launch and in several: one image, and each segment counted once
    scene = _scene(rt, "tilings", _abi.RT_LAMBERTIAN, 6)
    a = rt.Session(scene, seed=5, arithmetic="float64")
    b = rt.Session(scene, seed=5, arithmetic="float64", launch_seconds=1e-4)
    a.render_to(48)
    for passes in (16, 32, 48):
        b.render_to(passes)
    assert np.array_equal(a.pixels(), b.pixels())
    assert a.counters()["rays"] == b.counters()["rays"]
    # a plane of white under a white sky: a path's second segment leaves for good
    assert 160 * 120 * 48 < a.counters()["rays"] <= 2 * 160 * 120 * 48
