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
