"""The pool kernel (a session's AUTO form) against the wavefront's steps on a B200, through the C-ABI.

Both render the same samples through the same arithmetic, rounding included, and add them in the same order, so the
images and the counts are equal, with no tolerance. Sizes where the pool can go wrong: one sample; fewer samples than a
warp; images whose tiles hang over both edges (claimed numbers without a pixel); more samples than every warp's paths;
several launches; paths of one segment. Scenes: both searches, both integrators, with and without the second book's
features.
"""
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SCENES = [("weekend", {}), ("weekend", dict(combination="mis")), ("glass", {}), ("glass", dict(sampling="lights")),
          ("cornell-mis", {}), ("final", {}), ("bouncing", {}), ("smoke", {}), ("smoke", dict(combination="mis")),
          ("perlin", {}), ("light", dict(combination="mis")), ("ggx-furnace", {}),
          ("mesh-ggx", dict(mesh_level=3, env_width=64)), ("mesh-ggx", dict(mesh_level=6, env_width=64))]
SIZES = [(1, 1, 1, 0), (3, 5, 2, 0), (37, 21, 19, 0), (130, 67, 33, 0), (64, 64, 16, 1), (64, 64, 16, 2)]


BARE = [("quads", {}), ("materials", {}), ("furnace", {})]  # rendered by the persistent kernel otherwise


def _equal(rt, scene, seed, passes, form="wavefront", **kw):
    a = rt.Session(scene, seed=seed, **kw)
    b = rt.Session(scene, seed=seed, form=form, **kw)
    a.render_to(passes)
    b.render_to(passes)
    assert np.array_equal(a.pixels(), b.pixels())
    ca, cb = a.counters(), b.counters()
    assert (ca["rays"], ca["shadow_rays"]) == (cb["rays"], cb["shadow_rays"])


@pytest.mark.parametrize("name,kw", SCENES, ids=[f"{n}-{'-'.join(str(v) for v in k.values())}" for n, k in SCENES])
def test_pool_equals_the_wavefronts_steps(rt, name, kw):
    for width, height, passes, depth in SIZES:
        scene = rt.Scene(rt.builtin_scene(name, width=width, height=height, spp=passes, depth=depth, **kw))
        _equal(rt, scene, 11, passes)


@pytest.mark.parametrize("name,kw", BARE, ids=[n for n, _ in BARE])
def test_pool_equals_the_persistent_kernel_on_bare_scenes(rt, name, kw):
    for width, height, passes, depth in SIZES:
        scene = rt.Scene(rt.builtin_scene(name, width=width, height=height, spp=passes, depth=depth, **kw))
        _equal(rt, scene, 11, passes, form="persistent")


@pytest.mark.parametrize("name", ["weekend", "glass"])
def test_pool_many_samples_and_launches(rt, name):
    # 8.9M samples in three launches: every warp's paths are renewed many times
    scene = rt.Scene(rt.builtin_scene(name, width=521, height=357, spp=48))
    _equal(rt, scene, 3, 48, launch_seconds=1e-4)


@pytest.mark.parametrize("name,width,height,seed", [("perlin", 1000, 800, 5), ("final", 500, 500, 5)])
def test_pool_equals_the_steps_in_rare_samples(rt, name, width, height, seed):
    # a last bit in a large sphere's or a volume's distances changes one sample in tens of millions
    _equal(rt, rt.Scene(rt.builtin_scene(name, width=width, height=height, spp=64)), seed, 64)


@pytest.mark.parametrize("name,kw", [("mesh-ggx", dict(depth=8, mesh_level=4, env_width=64)), ("final", dict(depth=2))])
def test_forms_by_a_launchs_size(rt, name, kw):
    # a first launch of 7.7M samples by the pool kernel, the rest of 23M by the steps: one image
    scene = rt.Scene(rt.builtin_scene(name, width=800, height=600, spp=64, **kw))
    a = rt.Session(scene, seed=8, launch_seconds=0.5)
    assert a.render_to(16)["kernel_launches"] == 3
    assert a.render_to(64)["kernel_launches"] > 3
    b = rt.Session(scene, seed=8, form="wavefront")
    b.render_to(64)
    assert np.array_equal(a.pixels(), b.pixels())


@pytest.mark.parametrize("name", ["quads", "materials"])
@pytest.mark.parametrize("width,height", [(1, 1), (37, 21), (512, 512), (520, 512)])
def test_a_bare_scenes_single_passes(rt, name, width, height):
    # one pass (by the persistent kernel up to 2^18 samples), then the rest of a chunk and more: one image
    scene = rt.Scene(rt.builtin_scene(name, width=width, height=height, spp=36))
    a = rt.Session(scene, seed=4)
    b = rt.Session(scene, seed=4, form="persistent")
    for passes in (1, 2, 20, 36):
        a.render_to(passes)
        b.render_to(passes)
        assert np.array_equal(a.pixels(), b.pixels())
    assert a.counters()["rays"] == b.counters()["rays"]


def test_a_tuned_session_takes_the_steps(rt):
    scene = rt.Scene(rt.builtin_scene("weekend", width=64, spp=16))
    s = rt.Session(scene, seed=2)
    s.render_to(16)
    image, launches = s.pixels(), s.render_to(16)["launches"]
    assert launches == 0
    t = rt.Session(scene, seed=2)
    t.set_tuning({**t.tuning(), "slots": 1 << 19})
    assert t.render_to(16)["kernel_launches"] > 3
    assert np.array_equal(t.pixels(), image)


@pytest.mark.parametrize("passes", [1, 16, 33])
@pytest.mark.parametrize("named", [[("weekend", {}), ("cover-60", {}), ("weekend", dict(combination="mis")),
                                    ("glass", {}), ("cover-900", {})],
                                   [("bouncing", {}), ("smoke", {}), ("final", {})]], ids=["plain", "features"])
def test_batched_tree_jobs_equal_their_sessions(rt, named, passes):
    # books' jobs on trees, of sizes whose tiles hang over the edges and whose samples start anywhere in a claim,
    # between jobs of the other groups (NEE/MIS, flat-searched scenes)
    jobs = [(rt.builtin_scene(n, width=21 + 8 * k, height=13 + 7 * k, spp=passes, **kw), 40 + k, passes)
            for k, (n, kw) in enumerate(named)]
    batch = rt.batch_render(jobs)
    for (desc, seed, _), image, (name, kw) in zip(jobs, batch.images, named):
        if name in ("glass", "smoke") or kw:
            continue  # kernels of their own roundings
        session = rt.Session(rt.Scene(desc), seed=seed, form="wavefront")
        session.render_to(passes)
        assert np.array_equal(image, session.pixels()), name


@pytest.mark.parametrize("scenes", [[("weekend", {}), ("cover-60", {}), ("cover-700", {})],
                                    [("final", {}), ("bouncing", {})]], ids=["plain", "features"])
def test_continuous_servers_books_requests_equal_their_sessions(rt, scenes):
    # refined in batched steps, each to the end of a chunk, after a first pass of its own
    server = rt.Server(hbm_budget_bytes=1 << 30, step_seconds=0.001, continuous=1)
    held = []
    for k, (name, kw) in enumerate(scenes):
        desc = rt.builtin_scene(name, width=33 + 10 * k, height=29, spp=35, **kw)
        scene = rt.Scene(desc)
        held.append((desc, scene, server.submit(scene, desc.camera, 60 + k, 35)))
    while any(server.poll(i)["state"] != "done" for _, _, i in held):
        assert all(server.poll(i)["passes"] in (0, 1, 35) or server.poll(i)["passes"] % 16 == 0 for _, _, i in held)
        server.step()
    for k, (desc, scene, i) in enumerate(held):
        session = rt.Session(scene, seed=60 + k, form="wavefront")
        session.render_to(1)
        session.render_to(35)
        assert np.array_equal(server.fetch(i), session.pixels()), scenes[k]
    assert server.stats()["used_bytes"] == 0
    server.close()


def test_an_image_whose_samples_are_too_many_to_number_is_refused(rt):
    # a chunk of 16 passes of 16,400 x 16,400 pixels has 2^32 samples and more; one pass has not
    scene = rt.Scene(rt.builtin_scene("cornell", width=64, spp=16, depth=1))
    session = rt.Session(scene, seed=1)
    session.set_camera(rt.builtin_camera("cornell", width=16400, height=16400, spp=16, depth=1))
    with pytest.raises(rt.CapacityError):
        session.render_to(16)
    assert session.state() == 0


def test_a_bare_scenes_samples_beyond_the_budget(rt):
    # 16 passes of 3,901 x 2,201 pixels are more samples than 2 GiB hold: the persistent kernel's launch, of two kernels;
    # of 8 passes the pool kernel's, of three
    scene = rt.Scene(rt.builtin_scene("quads", width=64, spp=16, depth=2))
    camera = rt.builtin_camera("quads", width=3901, height=2201, spp=16, depth=2)
    images = []
    for form, targets, kernels in (("auto", [16], [2]), ("auto", [8, 16], [3, 3]), ("persistent", [16], [2])):
        session = rt.Session(scene, seed=1, form=form, launch_seconds=0.5)
        session.set_camera(camera)
        assert [session.render_to(t)["kernel_launches"] for t in targets] == kernels
        images.append(session.pixels() if len(targets) == 1 else None)
    assert np.array_equal(images[0], images[2])


@pytest.mark.parametrize("arithmetic", ["float32", "float64"])
def test_a_first_launch_of_long_paths_is_short(rt, arithmetic):
    # a white room without a way out: paths run to their 4,000th segment, and a launch is asked to take 50 ms
    import ctypes as C

    from raytracing_b200 import _abi

    def v(x, y, z):
        return _abi.Vec3(float(x), float(y), float(z))

    walls = []
    for a in range(3):
        for side in (-3, 3):
            q, u, w = [-3, -3, -3], [0, 0, 0], [0, 0, 0]
            q[a], u[(a + 1) % 3], w[(a + 2) % 3] = side, 6, 6
            walls.append(_abi.QuadDesc(q=v(*q), u=v(*u), v=v(*w)))
    quads, textures, materials = (_abi.QuadDesc * 6)(*walls), (_abi.TextureDesc * 1)(), (_abi.MaterialDesc * 1)()
    textures[0] = _abi.TextureDesc(kind=_abi.RT_TEXTURE_SOLID)
    textures[0].rgb = v(1, 1, 1)
    materials[0] = _abi.MaterialDesc(kind=_abi.RT_LAMBERTIAN, texture=0)
    cam = _abi.CameraDesc(image_width=64, image_height=64, sqrt_spp=1, max_depth=4000, center=v(0, 0, 2),
                          sampling=_abi.RT_SAMPLING_MATERIAL)
    cam.pixel_delta_u, cam.pixel_delta_v, cam.pixel00_loc = v(1 / 64, 0, 0), v(0, -1 / 64, 0), v(-0.5, 0.5, 1)
    desc = _abi.SceneDesc(quads=quads, quad_count=6, materials=materials, material_count=1, textures=textures,
                          texture_count=1, camera=cam)
    session = rt.Session(rt.Scene(C.pointer(desc)), seed=1, arithmetic=arithmetic, launch_seconds=0.05)
    report = session.render_to(512)
    assert session.counters()["rays"] > 1000 * 64 * 64 * 512  # (a ray leaves through an edge now and then)
    assert report["launches"] > 1 and report["longest_launch_seconds"] < 0.1


@pytest.mark.parametrize("passes", [1, 17])
def test_a_batched_tree_job_beside_others_with_features(rt, passes):
    # a step of few samples, plain scenes and scenes with motion, textures or smoke in one batch
    named = ["weekend", "final", "cover-700", "bouncing", "cover-2000"]
    jobs = [(rt.builtin_scene(n, width=160 + 8 * k, height=120, spp=passes), 70 + k, passes) for k, n in enumerate(named)]
    batch = rt.batch_render(jobs)
    for (desc, seed, _), image, name in zip(jobs, batch.images, named):
        session = rt.Session(rt.Scene(desc), seed=seed)
        session.render_to(passes)
        assert np.array_equal(image, session.pixels()), name


def _every_material(rt, shapes, moving):
    """Shapes at any angle under NEE with MIS, of every material, with lamps among them: matte, mirrors, glass, metal
    rough, smooth and below the roughness of a perfect mirror, a coat, lamps that are spheres and quads at any angle."""
    import ctypes as C

    from raytracing_b200 import _abi

    def v(p):
        return _abi.Vec3(*(float(x) for x in p))

    r = np.random.default_rng(shapes)
    kinds = [(_abi.RT_LAMBERTIAN, 0, 0), (_abi.RT_METAL, 0, 0), (_abi.RT_DIELECTRIC, 0, 0), (_abi.RT_DIFFUSE_LIGHT, 0, 0),
             (_abi.RT_METAL, _abi.RT_MICROFACET_CONDUCTOR, 0.4), (_abi.RT_METAL, _abi.RT_MICROFACET_CONDUCTOR, 0.02),
             (_abi.RT_LAMBERTIAN, _abi.RT_MICROFACET_GLOSS, 0.4)]
    n = len(kinds)
    textures, materials, facets = (_abi.TextureDesc * 2)(), (_abi.MaterialDesc * n)(), (_abi.MicrofacetDesc * n)()
    textures[0], textures[1] = _abi.TextureDesc(), _abi.TextureDesc()
    textures[0].rgb, textures[1].rgb = v((0.7, 0.6, 0.5)), v((5, 6, 4))
    for k, (kind, facet, roughness) in enumerate(kinds):
        materials[k] = _abi.MaterialDesc(kind=kind, texture=int(kind == _abi.RT_DIFFUSE_LIGHT), albedo=v((0.9, 0.7, 0.5)),
                                         refraction_index=1.5)
        facets[k] = _abi.MicrofacetDesc(kind=facet, roughness=roughness)
    s = (_abi.SphereDesc * shapes)(*[_abi.SphereDesc(center=v(r.uniform(-4, 4, 3)), radius=r.uniform(0.2, 1.0),
                                                     material=i % n, uv_cos=1.0) for i in range(shapes)])
    q = (_abi.QuadDesc * shapes)(*[_abi.QuadDesc(q=v(r.uniform(-5, 4, 3)), u=v(r.uniform(-2, 2, 3)),
                                                 v=v(r.uniform(-2, 2, 3)), material=i % n) for i in range(shapes)])
    if moving:
        s[0].displacement = v((0.3, 0.2, -0.1))
    cam = _abi.CameraDesc(image_width=64, image_height=48, sqrt_spp=4, max_depth=10, center=v((0, 0, 11)),
                          sampling=_abi.RT_SAMPLING_MATERIAL)
    cam.sky_bottom, cam.sky_top = v((0.3, 0.3, 0.3)), v((0.1, 0.2, 0.3))
    cam.pixel_delta_u, cam.pixel_delta_v = v((1 / 64, 0, 0)), v((0, -1 / 64, 0))
    cam.pixel00_loc = v((-0.5, 0.375, 10))
    desc = _abi.SceneDesc(spheres=s, sphere_count=shapes, quads=q, quad_count=shapes, materials=materials, material_count=n,
                          textures=textures, texture_count=2, microfacets=facets, microfacet_count=n, camera=cam,
                          combination=_abi.RT_COMBINE_POWER_HEURISTIC, quality=1)
    return rt.Scene(C.pointer(desc))


@pytest.mark.parametrize("moving", [False, True])
@pytest.mark.parametrize("shapes", [10, 60], ids=["flat", "tree"])
def test_every_material_under_nee(rt, shapes, moving):
    # the pool kernel, the steps, and the steps as they were before the pool kernel: one image, to the last bit
    scene = _every_material(rt, shapes, moving)
    assert scene.stats()["flat"] == (shapes == 10)
    _equal(rt, scene, 9, 16)
    session = rt.Session(scene, seed=9)
    session.render_to(16)
    want = np.load(Path(__file__).resolve().parent / "golden" / "nee_materials.npz")[f"{shapes}-{int(moving)}"]
    assert np.array_equal(session.pixels(), want)
