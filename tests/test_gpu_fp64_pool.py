"""The FP64 integrator's pool kernel on a B200, through the C-ABI, at the sizes where it can go wrong.

The image of N passes is the same bit for bit in one call and in calls of its parts (other launches, other warps and
lists), its segment count too: one sample; fewer samples than a warp; tiles over both edges; more samples than every
warp's paths; paths of one segment. The walk tests its boxes in float: a box it wrongly skipped would turn hits into
misses, which on paths of one segment (a miss is the sky, a hit black) moves the image's mean away from the float
render's, whose hits are checked against the oracle's (tests/test_gpu_render.py).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SCENES = ["weekend", "glass", "bouncing", "final", "smoke", "quads", "cover-900"]
SIZES = [(1, 1, 1, 0), (3, 5, 2, 0), (37, 21, 35, 0), (64, 64, 17, 1), (211, 97, 33, 0)]


@pytest.mark.parametrize("name", SCENES)
def test_passes_in_parts(rt, name):
    for width, height, passes, depth in SIZES:
        scene = rt.Scene(rt.builtin_scene(name, width=width, height=height, spp=passes, depth=depth))
        a = rt.Session(scene, seed=9, arithmetic="float64")
        a.render_to(passes)
        b = rt.Session(scene, seed=9, arithmetic="float64", launch_seconds=1e-4)
        for target in sorted({min(16, passes), min(32, passes), passes}):
            b.render_to(target)
        assert np.array_equal(a.pixels(), b.pixels()), (name, width, height)
        assert a.counters()["rays"] == b.counters()["rays"]


@pytest.mark.parametrize("name", ["weekend", "cover-900", "final", "materials"])
def test_one_segment_paths_agree_with_float(rt, name):
    # depth 1: a path's one ray leaves (sky), meets a lamp, or ends black; float and double see the same camera rays
    # but for their uniforms' last bits, so all but the pixels an edge passes through agree
    scene = rt.Scene(rt.builtin_scene(name, width=160, height=100, spp=16, depth=1))
    f, d = rt.Session(scene, seed=3), rt.Session(scene, seed=3, arithmetic="float64")
    f.render_to(16)
    d.render_to(16)
    assert abs(f.pixels().mean() - d.pixels().mean()) <= 5e-3 * max(d.pixels().mean(), 1e-3)


def _boxes_scene(rt, center, scale, seed, hidden):
    """24 matte spheres and quads, few enough to be searched one after another; with `hidden`, specks inside one of the
    spheres, which no ray reaches, make them a tree. Seen along an axis: the camera's middle rays have two directions
    of almost nothing."""
    import ctypes as C

    from raytracing_b200 import _abi

    def v(p):
        return _abi.Vec3(*(float(x) for x in p))

    r = np.random.default_rng(seed)
    at = np.array(center, dtype=float)
    place = at * [1, 1, 0]
    spheres = [_abi.SphereDesc(center=v(scale * r.uniform(-6, 6, 3) + place), radius=scale * r.uniform(0.2, 1.6), uv_cos=1.0)
               for _ in range(14)]
    quads = [_abi.QuadDesc(q=v(scale * r.uniform(-7, 3, 3) + place), u=v(scale * r.uniform(-4, 4, 3)),
                           v=v(scale * r.uniform(-4, 4, 3))) for _ in range(6)]
    quads += [_abi.QuadDesc(q=v(scale * np.array([8 * i - 8, 8 * j - 8, -7]) + place), u=v((8 * scale, 0, 0)),
                            v=v((0, 8 * scale, 0))) for i in range(2) for j in range(2)]
    if hidden:
        inside, radius = spheres[0].center, spheres[0].radius
        spheres += [_abi.SphereDesc(center=v(np.array([inside.x, inside.y, inside.z]) + radius * r.uniform(-0.3, 0.3, 3)),
                                    radius=radius * 0.01, uv_cos=1.0) for _ in range(30)]
    textures, materials = (_abi.TextureDesc * 1)(), (_abi.MaterialDesc * 1)()
    textures[0] = _abi.TextureDesc(kind=_abi.RT_TEXTURE_SOLID)
    textures[0].rgb = v((0.7, 0.6, 0.5))
    materials[0] = _abi.MaterialDesc(kind=_abi.RT_LAMBERTIAN, texture=0)
    cam = _abi.CameraDesc(image_width=201, image_height=151, sqrt_spp=4, max_depth=8, center=v(at),
                          sampling=_abi.RT_SAMPLING_MATERIAL)
    cam.sky_bottom, cam.sky_top = v((1, 1, 1)), v((0.5, 0.7, 1))
    step = 16 * scale / 201
    cam.pixel_delta_u, cam.pixel_delta_v = v((step, 0, 0)), v((0, -step, 0))
    cam.pixel00_loc = v((at[0] - 100 * step, at[1] + 75 * step, 0))
    s, q = (_abi.SphereDesc * len(spheres))(*spheres), (_abi.QuadDesc * len(quads))(*quads)
    desc = _abi.SceneDesc(spheres=s, sphere_count=len(spheres), quads=q, quad_count=len(quads), materials=materials,
                          material_count=1, textures=textures, texture_count=1, camera=cam)
    scene = rt.Scene(C.pointer(desc))
    assert scene.stats()["flat"] == (0 if hidden else 1)
    return scene


@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("center,scale", [((0, 0, 20), 1.0), ((0, 0, 3000), 1.0), ((4e4, -3e4, 2e5), 1.0), ((0, 0, 2e-2), 1e-3),
                                          ((500, 700, 20), 1.0)])
def test_the_float_boxes_miss_no_hit(rt, center, scale, seed):
    # every primitive tested in double, without a box, against the walk whose boxes are tested in float: the same image
    # and the same segments, bit for bit
    images = []
    for hidden in (False, True):
        session = rt.Session(_boxes_scene(rt, center, scale, seed, hidden), seed=3, arithmetic="float64")
        session.render_to(16)
        images.append((session.pixels(), session.counters()["rays"]))
    assert images[0][1] == images[1][1]
    assert np.array_equal(images[0][0], images[1][0])
    assert images[0][1] > 1.3 * 201 * 151 * 16  # paths that bounce


@pytest.mark.parametrize("name", ["quads", "weekend"])
def test_samples_beyond_the_budget_in_bands(rt, name):
    # 16 passes of 2,801 x 2,011 pixels are more samples than 2 GiB hold: two bands, whose last tiles hang over both
    # edges; of 8 passes one. The chunk's sums are added in two parts then: equal but for the rounding of 16 additions.
    scene = rt.Scene(rt.builtin_scene(name, width=64, spp=16, depth=2))
    camera = rt.builtin_camera(name, width=2801, height=2011, spp=16, depth=2)
    per_band = 4 if name == "weekend" else 3
    images, rays = [], []
    for targets, kernels in (([16], [2 * per_band]), ([8, 16], [per_band, per_band])):
        session = rt.Session(scene, seed=1, arithmetic="float64", launch_seconds=0.5)
        session.set_camera(camera)
        assert [session.render_to(t)["kernel_launches"] for t in targets] == kernels
        images.append(session.pixels())
        rays.append(session.counters()["rays"])
    assert rays[0] == rays[1]
    assert np.allclose(images[0], images[1], rtol=32 * 2.0 ** -53, atol=0)
