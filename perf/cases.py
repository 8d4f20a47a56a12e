"""The workloads whose speed this repository looks after, through its public Python handle.

Every case is a dict of plain values; "kind" says which call sequence it is:

  frame    one frame of the engine loop: gbr_shadow_pass + gbr_render_view
           (optionally with moved objects, normals, kernel3's switches, a
           pseudo-AA pass, or results in pinned host memory)
  graph    one replay of a captured batch of views with new cameras
  views    one uncaptured gbr_render_batch of views of uneven sizes
  served   one burst of requests through the serving loop, results in host memory
  post     the post passes over an already rendered frame

Scenes come from openclrenderer_gb300.scenes: the cubes, terrain, binning
stress, sphere and serving scenes of this repository's configurations.
"""
import math

import numpy as np
import torch

from openclrenderer_gb300 import scenes
from openclrenderer_gb300 import structs as S
from openclrenderer_gb300.pipeline import Batch, GpuScene, OutputSet, Server

FLAG_REFLECTIVE = 1  # FEATURE_FLAG_SS_REFLECTIVE
NO_TEXTURE = 0xFFFFFFFF


def listed():
    return [
        # The smallest frame: 768 triangles, one light, no cubemap.  A tool or
        # a preview window; launches and host work count.
        {"name": "cubes_800x600", "kind": "frame", "scene": "cubes", "width": 800, "height": 600},
        # The headline: one frame of a game over a million-triangle terrain,
        # 16 lights, 16 textures, a shadow cubemap rendered every frame.
        {"name": "terrain_1080p", "kind": "frame", "scene": "terrain", "nx": 1024, "nz": 512, "lights": 16,
         "shadows": 1, "width": 1920, "height": 1080},
        # The same frame delivered to pinned host memory (depth, id, colour),
        # as a caller without device buffers takes it.
        {"name": "terrain_1080p_host", "kind": "frame", "scene": "terrain", "nx": 1024, "nz": 512, "lights": 16,
         "shadows": 1, "width": 1920, "height": 1080, "host": True},
        # Heavy overdraw and dense small geometry: two million sub-pixel
        # triangles among a thousand screen-covering ones.
        {"name": "stress_1440p", "kind": "frame", "scene": "stress", "small": 2_000_000, "big": 1000,
         "width": 2560, "height": 1440},
        # The largest resolution over the largest serving scene.
        {"name": "serving_2m_4k", "kind": "frame", "scene": "serving", "triangles": 2_000_000, "width": 3840,
         "height": 2160},
        # A small scene whose objects move every frame (poses flushed, world
        # cache rebuilt), at an odd resolution, with normals and pseudo-AA.
        {"name": "moving_spheres_1279x721", "kind": "frame", "scene": "spheres", "spheres": 500, "lights": 8,
         "width": 1279, "height": 721, "moving": True, "normals": True, "aa": True},
        # Several shadow casters (one static too) and kernel3's optional
        # switches: normal maps and outlines.
        {"name": "shadows_features_1280x720", "kind": "frame", "scene": "serving", "triangles": 100_000,
         "shadows": 3, "features": True, "normals": True, "width": 1280, "height": 720},
        # Multi-camera rendering: 64 views of mixed size replayed as one graph.
        {"name": "spheres_graph_64", "kind": "graph", "scene": "spheres", "spheres": 500, "lights": 8, "views": 64},
        # A handful of views of ragged size in one plain call.
        {"name": "views_ragged_9", "kind": "views", "scene": "serving", "triangles": 500_000, "views": 9},
        # A burst of mixed requests on resident scenes (the serving loop).
        {"name": "served_burst_16", "kind": "served", "scenes": 4, "triangles": 2_000_000, "requests": 16},
        # The engine's post passes over a full-HD frame.
        {"name": "post_1080p", "kind": "post", "scene": "terrain", "nx": 1024, "nz": 512, "lights": 16, "shadows": 1,
         "width": 1920, "height": 1080},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _resolution(rng, hi=3840):
    """A width and a height between 160x120 and 4K, odd ones among them."""
    w = _log(rng, 160, hi)
    return w, max(90, min(2160, int(w * rng.uniform(0.5, 0.8))))


def draw(rng):
    kind = rng.choice(["cubes", "terrain", "terrain", "stress", "serving", "moving", "features", "graph", "views",
                       "served", "post"])
    if kind == "cubes":
        w, h = _resolution(rng)
        return {"kind": "frame", "scene": "cubes", "width": w, "height": h, "normals": rng.random() < 0.5}
    if kind in ("terrain", "post"):
        w, h = _resolution(rng)
        c = {"kind": "post" if kind == "post" else "frame", "scene": "terrain", "nx": 16 * _log(rng, 2, 64),
             "nz": _log(rng, 16, 512), "lights": rng.randint(1, 16), "shadows": rng.randint(0, 1), "width": w,
             "height": h}
        if kind == "terrain":
            c["host"] = rng.random() < 0.3
        return c
    if kind == "stress":
        w, h = _resolution(rng, 2560)
        return {"kind": "frame", "scene": "stress", "small": _log(rng, 20_000, 2_000_000), "big": _log(rng, 10, 1000),
                "width": w, "height": min(h, 1440)}
    if kind == "serving":
        w, h = _resolution(rng)
        return {"kind": "frame", "scene": "serving", "triangles": _log(rng, 100_000, 2_000_000), "width": w,
                "height": h}
    if kind == "moving":
        w, h = _resolution(rng, 1920)
        return {"kind": "frame", "scene": "spheres", "spheres": _log(rng, 20, 500), "lights": rng.randint(1, 8),
                "width": w, "height": h, "moving": True, "normals": True, "aa": rng.random() < 0.5}
    if kind == "features":
        w, h = _resolution(rng, 1920)
        return {"kind": "frame", "scene": "serving", "triangles": _log(rng, 100_000, 500_000),
                "shadows": rng.randint(2, 4), "features": True, "normals": rng.random() < 0.5, "width": w,
                "height": h}
    if kind == "graph":
        return {"kind": "graph", "scene": "spheres", "spheres": _log(rng, 50, 500), "lights": rng.randint(1, 8),
                "views": _log(rng, 2, 64)}
    if kind == "views":
        return {"kind": "views", "scene": "serving", "triangles": _log(rng, 100_000, 1_000_000),
                "views": rng.randint(2, 12)}
    return {"kind": "served", "scenes": rng.randint(1, 4), "triangles": _log(rng, 200_000, 2_000_000),
            "requests": rng.randint(2, 16)}


# ---- scenes -----------------------------------------------------------------------
def _scene(case, seed):
    kind = case["scene"]
    if kind == "cubes":
        return scenes.plain_cubes(seed=seed)
    if kind == "terrain":
        sc = scenes.terrain(seed=seed, nx=case["nx"], nz=case["nz"], width=case["width"], height=case["height"],
                            n_lights=case["lights"])
        sc.lights["shadow"] = np.arange(len(sc.lights)) < case["shadows"]
        return sc
    if kind == "stress":
        return scenes.binning_stress(n_small=case["small"], n_big=case["big"], width=case["width"],
                                     height=case["height"], seed=seed)
    if kind == "spheres":
        return scenes.spheres_batch(n_spheres=case["spheres"], n_views=case.get("views", 1), n_lights=case["lights"],
                                    seed=seed)
    sc = scenes.serving_scene(case["triangles"], seed=seed)
    if "shadows" in case:
        sc.lights["shadow"] = np.arange(len(sc.lights)) < case["shadows"]
        sc.lights["is_static"][1] = 1
    if case.get("features"):
        d = np.arange(len(sc.descs))
        sc.descs["rid"] = np.where(d % 2 == 0, (d + 3) % 8, NO_TEXTURE)
        sc.descs["feature_flag"] |= np.where(d % 3 == 0, S.FLAG_OUTLINE, 0).astype(np.int32)
        sc.descs["feature_flag"][8:40:4] |= S.FLAG_IS_STATIC
        sc.descs["feature_flag"][9:40:4] |= S.FLAG_NO_DYN_SHADOWS
    return sc


def _served_triangles(case):
    """Triangles of the resident scenes, the largest first: a full, a half, a quarter and a twentieth of the case's."""
    return [case["triangles"] // k for k in (1, 2, 4, 20)[:case["scenes"]]]


def _camera(case, sc, rng):
    """The scene's camera (serving: a random pose over the terrain), turned a little by the seed."""
    if case["scene"] == "serving":
        return scenes.random_pose(rng)
    cam = sc.cameras[0].copy()
    if case["scene"] != "stress":  # the stress scene is laid out in screen space
        cam["rot"][1] += rng.uniform(-0.2, 0.2)
    return cam


# The resolutions of a batch belong to the case; the poses to the seed.
def _graph_sizes(case):
    """The resolutions of a captured batch: the batched workload's mix."""
    rng = np.random.default_rng(case["views"])
    return [scenes.RESOLUTIONS_BATCH[rng.integers(0, len(scenes.RESOLUTIONS_BATCH))] for _ in range(case["views"])]


def _ragged_sizes(case):
    """The resolutions of an uncaptured batch: anything between a thumbnail and full HD."""
    rng = np.random.default_rng(case["views"])
    out = []
    for _ in range(case["views"]):
        w = int(round(math.exp(rng.uniform(math.log(160), math.log(1920)))))
        out.append((w, int(w * rng.uniform(0.5, 0.8))))
    return out


def _planes(sizes):
    """The outputs of many views, view after view in one buffer each for depth, id and colour."""
    total = sum(w * h for w, h in sizes)
    depth = torch.empty(total, dtype=torch.int32, device="cuda")
    ids, rgba = torch.empty_like(depth), torch.empty((total, 4), dtype=torch.uint8, device="cuda")
    outs, at = [], 0
    for w, h in sizes:
        o = OutputSet(1, 1)
        o.depth, o.id, o.rgba = (t[at:at + w * h].view(h, w, *t.shape[1:]) for t in (depth, ids, rgba))
        outs.append(o)
        at += w * h
    return [depth, ids, rgba], outs


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


# ---- what a program holds before the call ------------------------------------------
def prepare(case, seed):
    rng = np.random.default_rng(seed + 1000)
    if case["kind"] == "served":
        return _prepare_served(case, seed, rng)
    sc = _scene(case, seed)
    st = {"kind": case["kind"]}
    if case["kind"] == "post":
        return _prepare_post(case, sc, rng, st)
    g = st["gpu"] = GpuScene(sc)
    if case["kind"] == "graph":
        sizes = _graph_sizes(case)
        st["cams"] = sc.cameras
        st["planes"], outs = _planes(sizes)
        st["batch"] = Batch(g, [S.make_view(w, h, 90.0) for w, h in sizes], outs=outs)
        return st
    if case["kind"] == "views":
        sizes = _ragged_sizes(case)
        st["cams"] = [scenes.random_pose(rng) for _ in sizes]
        st["views"] = [S.make_view(w, h, 90.0) for w, h in sizes]
        st["outs"] = [OutputSet(w, h) for w, h in sizes]
        return st
    w, h = case["width"], case["height"]
    flags = S.VIEW_NORMAL_MAPPING | S.VIEW_OUTLINE if case.get("features") else 0
    st["cam"] = _camera(case, sc, rng)
    st["view"] = S.make_view(w, h, 90.0, flags=flags)
    if case.get("host"):
        st["host"] = [_pinned((h, w), torch.int32), _pinned((h, w), torch.int32), _pinned((h, w, 4), torch.uint8)]
        st["arrays"] = [st["host"][0].numpy().view(np.uint32), st["host"][1].numpy().view(np.uint32),
                        st["host"][2].numpy()]
    else:
        st["out"] = OutputSet(w, h, normals=bool(case.get("normals")))
    if case.get("aa"):
        st["aa"] = torch.empty_like(st["out"].rgba)
    if case.get("moving"):
        f = np.zeros(len(sc.descs), S.OBJECT_FLUSH)
        f["index"] = np.arange(len(sc.descs))
        for k in ("tid", "scale", "feature_flag"):
            f[k] = sc.descs[k]
        f["world_pos"] = sc.descs["world_pos"] + rng.uniform(-20, 20, (len(f), 4)) * (1, 1, 1, 0)
        q = rng.normal(size=(len(f), 4))
        f["world_rot_quat"] = q / np.linalg.norm(q, axis=1, keepdims=True)
        st["flush"] = f
    return st


def _prepare_served(case, seed, rng):
    st = {"kind": "served", "scenes": [GpuScene(scenes.serving_scene(n, seed=seed + i))
                                       for i, n in enumerate(_served_triangles(case))]}
    for g in st["scenes"]:
        g.shadow_pass()
    st["server"] = Server(st["scenes"])
    st["requests"] = []
    for i in range(case["requests"]):
        w, h = scenes.RESOLUTIONS_SERVE[(i // len(st["scenes"])) % len(scenes.RESOLUTIONS_SERVE)]
        rgba = _pinned((h, w, 4), torch.uint8)
        st["requests"].append((i % len(st["scenes"]), scenes.random_pose(rng), S.make_view(w, h, 90.0), rgba,
                               rgba.numpy()))
    return st


def _prepare_post(case, sc, rng, st):
    sc.descs["feature_flag"] |= np.where(np.arange(len(sc.descs)) % 2 == 0, FLAG_REFLECTIVE, 0).astype(np.int32)
    sc.lights["godray_intensity"][:2] = 0.5
    g = st["gpu"] = GpuScene(sc)
    st["cam"] = _camera(case, sc, rng)
    st["cam_old"] = st["cam"].copy()
    st["cam_old"]["pos"][:3] += rng.uniform(-10, 10, 3)
    st["cam_old"]["rot"][:2] += rng.uniform(-0.01, 0.01, 2)
    st["view"] = S.make_view(case["width"], case["height"], 90.0)
    g.shadow_pass()
    st["out"] = g.render(st["cam"], st["view"], normals=True)
    st["rgba"] = [torch.empty_like(st["out"].rgba) for _ in range(4)]
    return st


# ---- one pass ------------------------------------------------------------------------
class _Recoloured:
    """A rendered frame with the colours of a post pass: what the next pass reads."""

    def __init__(self, out, rgba):
        self.depth, self.id, self.normals, self.rgba = out.depth, out.id, out.normals, rgba


def run(state):
    kind = state["kind"]
    if kind == "graph":
        state["batch"].render(state["cams"])
        return state["planes"]
    if kind == "served":
        for i, (scene, cam, view, _, rgba) in enumerate(state["requests"]):
            state["server"].submit(scene, cam, view, rgba=rgba, tag=i)
        state["server"].drain()
        state["server"].poll()
        return [r[3] for r in state["requests"]]
    g = state["gpu"]
    if kind == "post":
        cam, view, out, r = state["cam"], state["view"], state["out"], state["rgba"]
        g.post_reflections(cam, view, out, rgba_out=r[0])
        g.post_godrays(cam, view, _Recoloured(out, r[0]), rgba_out=r[1])
        g.post_motion_blur(cam, state["cam_old"], view, _Recoloured(out, r[1]), frame_id=0, rgba_out=r[2])
        g.post_pseudo_aa(view, _Recoloured(out, r[2]), rgba_out=r[3])
        return r
    if "flush" in state:
        g.flush_objects(state["flush"])
    g.shadow_pass()
    if kind == "views":
        outs = g.render_batch(state["cams"], state["views"], outs=state["outs"])
        return [[o.depth, o.id, o.rgba] for o in outs]
    if "host" in state:
        a = state["arrays"]
        g.render_host(state["cam"], state["view"], depth=a[0], ids=a[1], rgba=a[2])
        return state["host"]
    o = g.render(state["cam"], state["view"], out=state["out"])
    outs = [o.depth, o.id, o.rgba]
    if o.normals is not None:
        outs.append(o.normals)
    if "aa" in state:
        outs.append(g.post_pseudo_aa(state["view"], o, rgba_out=state["aa"]))
    return outs


# ---- what a pass cannot do without ----------------------------------------------------
TRIANGLE_BYTES = 144   # one gbr_triangle, read once
PIXEL_BYTES = 12       # depth, id and RGBA8, written once
TEXEL_BYTES = 32       # the eight texels of a trilinear fetch (or the whole atlas, if that is less)
SETUP_FLOPS = 150      # transform, projection, edges and plane of a triangle on one surface
COVER_FLOPS = 20       # coverage and depth of a pixel
SHADE_FLOPS = 800      # kernel3 without its light loop: position, barycentrics, texture, occlusion
LIGHT_FLOPS = 60       # one light at one pixel
FACE_TEXELS = 6 * 1024 * 1024


def _triangles(case):
    return {"cubes": lambda: 768, "terrain": lambda: 2 * case["nx"] * case["nz"],
            "stress": lambda: case["small"] + case["big"], "spheres": lambda: 1000 * case["spheres"],
            "serving": lambda: case["triangles"]}[case["scene"]]()


def _lights(case):
    return {"cubes": 1, "stress": 4, "serving": 8}.get(case["scene"], case.get("lights", 8))


def _view_work(pixels, triangles, lights, views=1):
    return (PIXEL_BYTES + TEXEL_BYTES) * pixels + TRIANGLE_BYTES * triangles, \
        (SHADE_FLOPS + COVER_FLOPS + LIGHT_FLOPS * lights) * pixels + SETUP_FLOPS * triangles * views


def work(case):
    if case["kind"] == "served":
        tris = _served_triangles(case)
        n = len(tris)
        b = f = 0
        for i in range(case["requests"]):
            w, h = scenes.RESOLUTIONS_SERVE[(i // n) % len(scenes.RESOLUTIONS_SERVE)]
            bi, fi = _view_work(w * h, tris[i % n], 8)
            b, f = b + bi - (TRIANGLE_BYTES * tris[i % n] if i >= n else 0), f + fi
        return {"bytes": b, "flops": f}
    tris, lights = _triangles(case), _lights(case)
    if case["kind"] == "graph":
        pixels = sum(w * h for w, h in _graph_sizes(case))
        b, f = _view_work(pixels, tris, lights, case["views"])
        return {"bytes": b, "flops": f}
    if case["kind"] == "views":
        pixels = sum(w * h for w, h in _ragged_sizes(case))
        b, f = _view_work(pixels, tris, lights, case["views"])
        return {"bytes": b + 4 * FACE_TEXELS, "flops": f + SETUP_FLOPS * tris}
    pixels = case["width"] * case["height"]
    if case["kind"] == "post":  # 4 images read and written, depth / id / normals read, marches of some 80 taps
        return {"bytes": pixels * (4 * 8 + 12), "flops": pixels * 2000}
    b, f = _view_work(pixels, tris, lights)
    shadows = case.get("shadows", 1 if case["scene"] == "serving" else 0)
    if case["scene"] == "stress":  # every big triangle covers every pixel at its own depth
        f += COVER_FLOPS * pixels
    extra = 4 * pixels * (bool(case.get("normals")) + 2 * bool(case.get("aa")))
    return {"bytes": b + extra + 4 * FACE_TEXELS * shadows, "flops": f + SETUP_FLOPS * tris * shadows}


def exact(case, seed):
    """Every output is whole: quantised depths, triangle ids, RGBA8 bytes and
    16-bit normal codes, which stay equal, so none has a 64-bit value."""
    return None
