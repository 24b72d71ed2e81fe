"""Images and rays between the caller's memory and a B200, in blocks moved by several threads, through the C-ABI.

A query's hits do not depend on how its rays were cut into blocks: counts around a block's 16,384 rays and of several
blocks equal the same rays asked for a few at a time. An image's values are its sums times 1 / passes (a furnace's are
exactly 1), whatever its size: an odd number of values, around a block's 131,072 and several blocks. Calls from several
threads at once give what they give alone.
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rays(n, seed):
    r = np.random.default_rng(seed)
    o = np.array([13.0, 2.0, 3.0]) + r.uniform(-0.5, 0.5, (n, 3))
    return o.astype(np.float32), (r.uniform(-4, 4, (n, 3)) * [1, 0.2, 1] - o).astype(np.float32)


@pytest.mark.parametrize("n", [1, 16383, 16384, 16385, 40001, 300007])
def test_hits_do_not_depend_on_the_blocks(rt, n):
    scene = rt.Scene(rt.builtin_scene("weekend"))
    o, d = _rays(n, n)
    ids, ts = scene.closest_hits(o, d)
    parts = [scene.closest_hits(o[k:k + 7000], d[k:k + 7000]) for k in range(0, n, 7000)]
    assert np.array_equal(ids, np.concatenate([p[0] for p in parts]))
    assert np.array_equal(ts, np.concatenate([p[1] for p in parts]))
    assert (ids >= 0).any()


@pytest.mark.parametrize("width,height", [(1, 1), (5, 7), (209, 209), (211, 207), (640, 411)])
def test_images_of_any_size(rt, width, height):
    scene = rt.Scene(rt.builtin_scene("furnace", width=width, height=height, spp=3))
    session = rt.Session(scene, seed=1)
    session.render_to(3)
    assert np.array_equal(session.pixels(), np.ones((height, width, 3)))


def test_calls_from_several_threads(rt):
    scene = rt.Scene(rt.builtin_scene("weekend", width=400, spp=2))
    o, d = _rays(60001, 4)
    alone = scene.closest_hits(o, d)
    sessions = [rt.Session(scene, seed=k) for k in range(4)]
    for s in sessions:
        s.render_to(2)
    images = [s.pixels() for s in sessions]
    wrong = []

    def work(k):
        for _ in range(5):
            ids, ts = scene.closest_hits(o, d)
            if not (np.array_equal(ids, alone[0]) and np.array_equal(ts, alone[1])):
                wrong.append(k)
            if not np.array_equal(sessions[k].pixels(), images[k]):
                wrong.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.parametrize("name,kw", [("weekend", {}), ("cover-2000", {}), ("final", {}), ("mesh-ggx", dict(mesh_level=4)),
                                     ("glass", {})])
def test_a_ray_alone_and_among_others(rt, name, kw):
    # the four-wide walk's hits are checked against the oracle's in tests/test_gpu_render.py; a ray asked for alone
    # gives what it gives among its neighbours, whose walks share its warp
    scene = rt.Scene(rt.builtin_scene(name, width=64, height=36, **kw))
    o, d = scene.camera_rays(7, 0)
    ids, ts = scene.closest_hits(o, d)
    for k in range(0, len(o), 97):
        i, t = scene.closest_hits(o[k:k + 1], d[k:k + 1])
        assert i[0] == ids[k] and t[0] == ts[k]


@pytest.mark.parametrize("n", [100, 2000003])
def test_hits_over_the_rays_memory(rt, n):
    # a caller that needs its rays no more: the answers over the end of the origins and of the directions
    import ctypes as C

    scene = rt.Scene(rt.builtin_scene("weekend"))
    o, d = _rays(n, 8)
    ids, ts = scene.closest_hits(o, d)
    ts_over, ids_over = o.ravel()[2 * n:], d.ravel()[2 * n:].view(np.int32)
    p = lambda a, t: a.ctypes.data_as(C.POINTER(t))  # noqa: E731
    rt._check(rt._lib().rt_scene_closest_hits(scene._handle, p(o, C.c_float), p(d, C.c_float), n, p(ids_over, C.c_int32),
                                              p(ts_over, C.c_float)))
    assert np.array_equal(ts_over, ts)
    assert np.array_equal(ids_over, ids)
