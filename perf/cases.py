"""The framework's performance cases: what programs call it for, through its public entry points, from the smallest call
to the largest. A case is a dict of plain values; `listed()` names the fixed ones, `draw()` makes more of the same
ranges, `prepare()` what a program holds before the call, `run()` one pass of the call, `work()` the bytes and
operations it cannot do without, `exact()` the 64-bit answer where there is one.

Kinds of case (the "kind" of a case):
  hits     Scene.closest_hits: rays on the host in, primitive ids and distances out (picking, visibility queries)
  frame    a viewer's frame: Session.set_camera, render_to a few passes, display's bytes
  render   render(): scene tables on the host in, the finished image out, nothing kept between calls
  session  a long render on a resident scene: Session.set_camera, render_to, pixels
  batch    batch_render: many independent jobs of mixed sizes in one call
  serve    Server: requests of mixed scenes, sizes and targets submitted, stepped until done, fetched
"""
import math

import numpy as np
import torch

import raytracing_b200 as rt

# Scenes by what their kernels are: flat-searched or tree-searched, plain materials or the second book's features
# (textures, motion, smoke), the books' estimators or NEE with MIS, triangles with an environment map. With each, the
# mean path segments a sample takes (shadow rays included), measured once: a property of the scene, for work().
SEGMENTS = {
    "materials": 2.0, "quads": 1.6, "weekend": 2.6, "bouncing": 2.6, "checker": 1.9, "perlin": 1.9, "light": 3.0,
    "glass": 4.6, "cornell": 2.5, "smoke": 5.0, "final": 4.0, "cornell-mis": 10.6, "mesh-ggx": 3.0, "cover": 2.6,
}
PLAIN = ["materials", "quads", "weekend", "glass", "cornell", "cornell-mis", "light"]
FEATURES = ["bouncing", "checker", "perlin", "smoke", "final"]


def listed():
    return [
        # One ray: picking the object under a cursor; launch and copy latency, nothing else
        {"name": "pick_1", "kind": "hits", "scene": "weekend", "rays": 1, "spread": 1.0},
        # A frame's worth of visibility rays against the 1.3M-triangle mesh (an ordinary query batch, ragged size)
        {"name": "hits_mesh_230k", "kind": "hits", "scene": "mesh-ggx", "rays": 230401, "spread": 0.3, "level": 8},
        # The first frame of a moved camera in a viewer: one pass, then the screen's bytes
        {"name": "frame_weekend_256", "kind": "frame", "scene": "weekend", "width": 256, "height": 256, "passes": 1,
         "depth": 50, "tone": "books"},
        # The first book's cover through the one-shot call at its stated size (400x225, 32 passes, depth 50), in the
        # float and the double integrator
        {"name": "render_weekend_f32", "kind": "render", "scene": "weekend", "width": 400, "height": 225,
         "passes": 32, "depth": 50, "arithmetic": "float32"},
        {"name": "render_weekend_f64", "kind": "render", "scene": "weekend", "width": 400, "height": 225,
         "passes": 32, "depth": 50, "arithmetic": "float64"},
        # A small scene of a few bare shapes under the sky, an odd size
        {"name": "session_quads_397", "kind": "session", "scene": "quads", "width": 397, "height": 401, "passes": 100,
         "depth": 50},
        # The headline workload: the Cornell box with a glass ball under the books' mixture, 600x600 at 1024 passes
        {"name": "session_glass_600", "kind": "session", "scene": "glass", "width": 600, "height": 600,
         "passes": 1024, "depth": 50},
        # The same box under next-event estimation with multiple importance sampling
        {"name": "session_mis_600", "kind": "session", "scene": "cornell-mis", "width": 600, "height": 600,
         "passes": 256, "depth": 50},
        # The second book's final scene: textures, motion, smoke, a tree of a thousand boxes
        {"name": "session_final_400", "kind": "session", "scene": "final", "width": 400, "height": 400, "passes": 100,
         "depth": 40},
        # The 1.3M-triangle mesh, GGX, environment map, at full HD
        {"name": "session_mesh_1080p", "kind": "session", "scene": "mesh-ggx", "width": 1920, "height": 1080,
         "passes": 64, "depth": 16, "level": 8},
        # Independent jobs of uneven size in one call (cover variants of 50 to 2000 spheres)
        {"name": "batch_16", "kind": "batch", "jobs": 16, "largest": 512, "passes": 256},
        # A burst of requests served to completion: three resident scenes, mixed sizes and targets
        {"name": "serve_24", "kind": "serve", "requests": 24, "largest": 1024, "passes": 64, "continuous": 1},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["hits", "frame", "render", "session", "session", "session", "batch", "serve"])
    if kind == "hits":
        mesh = rng.random() < 0.5
        return {"kind": "hits", "scene": "mesh-ggx" if mesh else "weekend", "rays": _log_int(rng, 1, 400000),
                "spread": round(rng.uniform(0.1, 1.0), 3), **({"level": rng.randint(4, 8)} if mesh else {})}
    if kind == "frame":
        return {"kind": "frame", "scene": rng.choice(PLAIN + FEATURES), "width": _log_int(rng, 64, 1280),
                "height": _log_int(rng, 64, 720), "passes": _log_int(rng, 1, 8), "depth": _log_int(rng, 4, 50),
                "tone": rng.choice(["books", "agx", "neutral"])}
    if kind == "render":
        double = rng.random() < 0.4
        return {"kind": "render", "scene": rng.choice(["weekend", "glass", "materials", "perlin", "smoke"]),
                "width": _log_int(rng, 40, 500), "height": _log_int(rng, 40, 400), "passes": _log_int(rng, 1, 64),
                "depth": _log_int(rng, 4, 50), "arithmetic": "float64" if double else "float32"}
    if kind == "session":
        scene = rng.choice(PLAIN + FEATURES + ["mesh-ggx"] * 3)
        width, height = _log_int(rng, 100, 1400), _log_int(rng, 100, 1000)
        passes = _log_int(rng, 8, max(16, min(1024, 60_000_000 // (width * height))))
        return {"kind": "session", "scene": scene, "width": width, "height": height, "passes": passes,
                "depth": _log_int(rng, 4, 50), **({"level": rng.randint(5, 8)} if scene == "mesh-ggx" else {})}
    if kind == "batch":
        return {"kind": "batch", "jobs": _log_int(rng, 2, 24), "largest": _log_int(rng, 128, 512),
                "passes": _log_int(rng, 17, 256)}
    return {"kind": "serve", "requests": _log_int(rng, 2, 24), "largest": _log_int(rng, 128, 1024),
            "passes": _log_int(rng, 4, 64), "continuous": rng.choice([0, 1])}


_SCENES = {}  # a program makes a resident scene once and renders many views of it


def _description(name, case):
    extra = {"mesh_level": case["level"]} if "level" in case else {}
    return rt.builtin_scene(name, width=case.get("width", 0), height=case.get("height", 0),
                            spp=case.get("passes", 0), depth=case.get("depth", 0), **extra)


def _resident(name, case):
    key = (name, case.get("level"))
    if key not in _SCENES:
        _SCENES[key] = rt.Scene(rt.builtin_scene(name, **({"mesh_level": case["level"]} if "level" in case else {})))
    return _SCENES[key]


def _pick_rays(case, seed):
    """Rays toward the scene from around the camera: the origins jittered, the directions spread over the view."""
    r = np.random.default_rng(seed)
    n = case["rays"]
    center = np.array([13.0, 2.0, 3.0]) if case["scene"] == "weekend" else np.array([0.0, 2.0, 9.0])
    origins = center + r.uniform(-0.5, 0.5, (n, 3))
    targets = r.uniform(-1.0, 1.0, (n, 3)) * np.array([6.0, 1.2, 6.0]) * case["spread"]
    return origins.astype(np.float32), (targets - origins).astype(np.float32)


def _batch_jobs(case, seed):
    """Job sizes fixed by the case (so that every seed costs the same), contents by the seed."""
    sizes = np.random.default_rng(1000 + case["jobs"] + case["passes"])
    jobs = []
    for k in range(case["jobs"]):
        w, h = (int(round(math.exp(sizes.uniform(math.log(64), math.log(case["largest"]))))) for _ in range(2))
        passes = int(round(math.exp(sizes.uniform(math.log(16), math.log(case["passes"])))))
        spheres = int(round(math.exp(sizes.uniform(math.log(50), math.log(2000)))))
        jobs.append((w, h, passes, spheres, seed * 64 + k))
    return jobs


SERVED = ["weekend", "glass", "mesh-ggx"]


def _requests(case):
    sizes = np.random.default_rng(2000 + case["requests"] + case["largest"])
    out = []
    for k in range(case["requests"]):
        w = int(round(math.exp(sizes.uniform(math.log(100), math.log(case["largest"])))))
        h = max(64, int(w * sizes.uniform(0.5, 1.0)))
        passes = int(round(math.exp(sizes.uniform(0.0, math.log(case["passes"])))))
        orbit = (float(sizes.uniform(0, 360)), float(sizes.uniform(5, 40)))
        out.append((SERVED[k % 3], w, h, passes, orbit))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "hits":
        origins, directions = _pick_rays(case, seed)
        return {"case": case, "scene": _resident(case["scene"], case), "o": origins, "d": directions}
    if kind == "render":
        desc = _description(case["scene"], case)
        return {"case": case, "desc": desc, "seed": seed}
    if kind in ("frame", "session"):
        scene = _resident(case["scene"], case)
        return {"case": case, "session": rt.Session(scene, seed=seed),
                "camera": rt.builtin_camera(case["scene"], width=case["width"], height=case["height"],
                                            spp=case["passes"], depth=case["depth"])}
    if kind == "batch":
        jobs = [(rt.builtin_scene("cover-%d" % n, width=w, height=h, spp=p, scene_seed=s), s, p)
                for w, h, p, n, s in _batch_jobs(case, seed)]
        return {"case": case, "jobs": jobs}
    scenes = {name: _resident(name, {"level": 7} if name == "mesh-ggx" else {}) for name in SERVED}
    requests = [(scenes[name], rt.builtin_camera(name, width=w, height=h, spp=passes, orbit=orbit), seed * 64 + k, passes)
                for k, (name, w, h, passes, orbit) in enumerate(_requests(case))]
    return {"case": case, "requests": requests,
            "server": rt.Server(hbm_budget_bytes=8 << 30, continuous=case["continuous"])}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "hits":
        ids, ts = state["scene"].closest_hits(state["o"], state["d"])
        return {"ids": ids, "ts": ts}
    if kind == "render":
        r = rt.render(state["desc"], seed=state["seed"], passes=case["passes"], arithmetic=case["arithmetic"])
        return {"pixels": r.pixels, "rays": r.rays}
    if kind == "frame":
        s = state["session"]
        s.set_camera(state["camera"])
        s.render_to(case["passes"])
        return {"rgba": s.display(case["tone"])}
    if kind == "session":
        s = state["session"]
        s.set_camera(state["camera"])
        s.render_to(case["passes"])
        return {"pixels": s.pixels()}
    if kind == "batch":
        return {"images": rt.batch_render(state["jobs"]).images}
    server = state["server"]
    ids = [server.submit(scene, camera, seed, passes) for scene, camera, seed, passes in state["requests"]]
    while True:
        report = server.step()
        if report["active"] == 0 and report["queued"] == 0:
            break
    return {"images": [server.fetch(i) for i in ids]}


def _path_work(samples, pixels, scene):
    """A sample's segments, each a search (about log2 of the primitives, or all of a small scene) and a vertex's
    shading: some 400 operations; the image's sums written once, 24 bytes a pixel."""
    return 24.0 * pixels, 400.0 * SEGMENTS[scene] * samples


def work(case):
    kind = case["kind"]
    if kind == "hits":
        return {"bytes": 32.0 * case["rays"], "flops": 400.0 * case["rays"]}
    parts = []
    if kind in ("frame", "render", "session"):
        pixels = case["width"] * case["height"]
        parts = [(pixels * case["passes"], pixels, case["scene"])]
    elif kind == "batch":
        parts = [(w * h * p, w * h, "cover") for w, h, p, _, _ in _batch_jobs(case, 0)]
    else:
        parts = [(w * h * p, w * h, name) for name, w, h, p, _ in _requests(case)]
    totals = [_path_work(*p) for p in parts]
    return {"bytes": sum(t[0] for t in totals), "flops": sum(t[1] for t in totals)}


def exact(case, seed):
    """The distances of the rays' hits on the cover scene in 64 bits, every sphere tested (the quadratic of each, its
    nearest root beyond 0.001). A Monte Carlo image has no such value: its paths are the float ones' own, and a 64-bit
    walk leaves them at the first branch a rounding decides; nor has a ray against a million triangles in this time."""
    if case["kind"] != "hits" or case["scene"] != "weekend":
        return None
    owned = rt.builtin_scene("weekend")
    desc = owned.desc.contents
    spheres = np.array([[s.center.x, s.center.y, s.center.z, s.radius]
                        for s in (desc.spheres[i] for i in range(desc.sphere_count))])
    o, d = (torch.from_numpy(v.astype(np.float64)) for v in _pick_rays(case, seed))
    c, r = torch.from_numpy(spheres[:, :3]), torch.from_numpy(spheres[:, 3])
    out = []
    for at in range(0, o.shape[0], 4096):
        oo, dd = o[at:at + 4096, None, :], d[at:at + 4096, None, :]
        oc = c[None] - oo
        a = (dd * dd).sum(-1)
        h = (dd * oc).sum(-1) / a
        rest = oc - h[..., None] * dd
        disc = r * r - (rest * rest).sum(-1)
        half = torch.sqrt(disc.clamp(min=0.0) / a)
        near, far = h - half, h + half
        t = torch.where(near > 0.001, near, far)
        t = torch.where((disc >= 0) & (t > 0.001), t, torch.full_like(t, math.inf))
        out.append(t.min(dim=1).values)
    return {"ids": None, "ts": torch.cat(out)}
