"""Timed cases of the path tracer: whole render calls through its public entry points.

Each case is one call as a host program makes it (the add-on's viewport, material
previews and F12 renders, the request loop's batches, a converged reference, a
scene push), on this repository's own scenes (lucid_scenes.py) at the sizes its
tests and benchmark use.  Scenes, sample offsets and the camera are made from
the seed, so another seed is another picture.

Guided renders are not here: the guide trains on records taken in arrival order,
so two runs of the same call give images that differ by their noise.
"""
import math
import os
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "blender-lucid-renderer_b200"))
import lucid_capi  # noqa: E402
import lucid_scenes as ls  # noqa: E402

# Mean path segments per sample (closest-hit queries) of each scene, for work().
SEGMENTS = {"cornell": 3.2, "preview": 2.0, "hard_indirect": 4.0, "all_lights": 1.75, "textured": 1.4,
            "procedural": 2.0}

# Triangles of a procedural scene by icosphere level: 200 objects, the ground, two emitters, a volume box.
PROCEDURAL_LEVELS = {2: 66_574, 3: 258_574, 4: 1_026_574}


def listed():
    return [
        # the first, coarse answer of a viewport after a change: one call's latency
        {"name": "viewport_96x64", "entry": "render", "scene": "cornell", "tris": 36, "algo": "mis",
         "w": 96, "h": 64, "spp": 1, "depth": 8},
        # one tick of an 800x600 viewport session: one sample a pixel, the picture stays on the device
        {"name": "viewport_800x600", "entry": "device", "scene": "cornell", "tris": 36, "algo": "mis",
         "w": 800, "h": 600, "spp": 1, "depth": 8},
        # a draw callback that must not allocate: every light type, glass and metal
        {"name": "noalloc_203x127_4spp", "entry": "noalloc", "scene": "all_lights", "tris": 667, "algo": "mis",
         "w": 203, "h": 127, "spp": 4, "depth": 8},
        # a material preview thumbnail at its final quality
        {"name": "preview_256x256_32spp", "entry": "render", "scene": "preview", "tris": 5122, "algo": "mis",
         "w": 256, "h": 256, "spp": 32, "depth": 8},
        # a ragged frame with participating media and every light type
        {"name": "volume_333x207_5spp", "entry": "render", "scene": "all_lights", "tris": 667, "algo": "volume_mis",
         "w": 333, "h": 207, "spp": 5, "depth": 16},
        # node-graph materials under next-event estimation
        {"name": "textured_640x360_8spp", "entry": "render", "scene": "textured", "tris": 20, "algo": "nee",
         "w": 640, "h": 360, "spp": 8, "depth": 8},
        # an interior lit indirectly, the first iteration of an F12 render (4 samples)
        {"name": "interior_1280x720_4spp", "entry": "device", "scene": "hard_indirect", "tris": 20828, "algo": "mis",
         "w": 1280, "h": 720, "spp": 4, "depth": 8},
        # many small jobs on scenes of their own, in one call
        {"name": "batch_12_jobs", "entry": "batch", "scene": "cornell", "tris": 20_000, "algo": "mis",
         "w": 160, "h": 128, "spp": 8, "depth": 8, "jobs": 12},
        # an FP64-accumulated reference on a tessellated room
        {"name": "reference_f64_128x128_256spp", "entry": "f64", "scene": "cornell", "tris": 100_000, "algo": "simple",
         "w": 128, "h": 128, "spp": 256, "depth": 8},
        # a scene push as every edit in the add-on makes it, and its first frame
        {"name": "load_258k_tris", "entry": "load", "scene": "procedural", "tris": 258_574, "algo": "volume_mis",
         "w": 320, "h": 180, "spp": 1, "depth": 16},
        # the first iteration of the benchmark frame's F12 render, without media
        {"name": "f12_1M_960x540_4spp", "entry": "render", "scene": "procedural", "tris": 1_026_574, "algo": "mis",
         "w": 960, "h": 540, "spp": 4, "depth": 16},
        # the benchmark frame: 1M triangles, 1080p, 64 samples, media
        {"name": "f12_1M_1920x1080_64spp", "entry": "render", "scene": "procedural", "tris": 1_026_574,
         "algo": "volume_mis", "w": 1920, "h": 1080, "spp": 64, "depth": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _tris(kind, rng):
    fixed = {"preview": 5122, "hard_indirect": 20828, "all_lights": 667, "textured": 20}
    return fixed.get(kind) or _log(rng, 36, 500_000)


def draw(rng):
    entry = rng.choice(["render", "render", "render", "device", "device", "noalloc", "batch", "f64", "load"])
    c = {"entry": entry, "depth": rng.choice([4, 8, 8, 16])}
    if entry == "batch":
        return dict(c, scene="cornell", tris=_log(rng, 36, 100_000), algo=rng.choice(["nee", "mis", "volume_mis"]),
                    w=_log(rng, 48, 320), h=_log(rng, 48, 320), spp=_log(rng, 1, 16), jobs=rng.randint(4, 16))
    if entry == "load":
        level = rng.choice([2, 3])
        return dict(c, scene="procedural", tris=PROCEDURAL_LEVELS[level], algo=rng.choice(["mis", "volume_mis"]),
                    w=_log(rng, 64, 640), h=_log(rng, 64, 360), spp=1)
    if entry == "noalloc":
        kind = rng.choice(["cornell", "preview", "all_lights"])
        return dict(c, scene=kind, tris=_tris(kind, rng),
                    algo=rng.choice(["nee", "mis", "volume_mis"]), w=_log(rng, 32, 256), h=_log(rng, 32, 256),
                    spp=_log(rng, 1, 16))
    c["scene"] = rng.choice(["cornell", "preview", "hard_indirect", "all_lights", "textured", "procedural"])
    c["algo"] = rng.choice(["simple", "nee", "mis", "mis", "volume_simple", "volume_mis", "volume_mis"])
    c["tris"] = PROCEDURAL_LEVELS[rng.choice([2, 3, 4])] if c["scene"] == "procedural" else _tris(c["scene"], rng)
    if entry == "f64":
        return dict(c, w=_log(rng, 32, 320), h=_log(rng, 32, 200), spp=_log(rng, 16, 256))
    c["w"] = _log(rng, 48, 1920)
    c["h"] = max(32, min(1080, round(c["w"] / rng.uniform(0.8, 2.0))))
    return dict(c, spp=_log(rng, 1, max(1, min(64, 24_000_000 // (c["w"] * c["h"])))))


def _scene(case, seed):
    """(scene dict, camera) of the case from the seed; the camera moves a little with it."""
    kind = case["scene"]
    if kind == "cornell":
        scene, cam = ls.cornell_variant(seed, case["tris"])
    elif kind == "preview":
        scene, cam = ls.material_preview_scene(seed)
    elif kind == "hard_indirect":
        scene, cam = ls.hard_indirect_scene()
    elif kind == "textured":
        scene, cam = ls.textured_scene()
    elif kind == "all_lights":
        scene, cam = ls.all_lights_scene(tempfile.gettempdir())
    else:
        level = next(k for k, n in PROCEDURAL_LEVELS.items() if n == case["tris"])
        scene, cam = ls.procedural_scene(seed=seed % 100_003, levels=level, workdir=tempfile.gettempdir())
    rng = np.random.default_rng(seed)
    cam = [float(x) for x in cam]
    cam[0:6] = [c + float(e) for c, e in zip(cam[0:6], rng.uniform(-0.02, 0.02, 6))]
    return scene, tuple(cam)


def _context(case, seed):
    """A context with the case's scene, camera and integrator."""
    scene, cam = _scene(case, seed)
    ctx = lucid_capi.Context(0)
    if case["scene"] == "textured":
        ctx.load_scene_json(ls.to_json(scene))   # node graphs come as JSON
    else:
        ctx.load_scene_arrays(ls.scene_arrays(scene, json_rounding=False))
    ctx.set_camera(*cam)
    ctx.set_algorithm(case["algo"])
    return ctx, cam


def prepare(case, seed):
    s = {"case": case, "offset": int(np.random.default_rng(seed + 1).integers(0, 1 << 20))}
    w, h = case["w"], case["h"]
    if case["entry"] == "load":
        scene, s["cam"] = _scene(case, seed)
        s["arrays"] = ls.scene_arrays(scene, json_rounding=False)
        s["ctx"] = lucid_capi.Context(0)
        s["ctx"].set_algorithm(case["algo"])
    elif case["entry"] == "batch":
        s["ctx"] = lucid_capi.Context(0)
        s["jobs"] = []
        for k in range(case["jobs"]):   # sizes and samples around the case's, each job on a scene of its own
            ctx, cam = _context(dict(case, tris=max(36, case["tris"] * (1 + k % 3) // 2)), seed * 64 + k)
            s["jobs"].append({"scene": ctx, "camera": cam, "width": max(8, w + 16 * (k % 4) - 5 * (k % 2)),
                              "height": max(8, h - 7 * (k % 3)), "samples": max(1, case["spp"] >> (k % 3)),
                              "sample_offset": s["offset"], "max_depth": case["depth"]})
    else:
        s["ctx"], _ = _context(case, seed)
    if case["entry"] in ("device", "noalloc"):
        s["out"] = torch.empty((h, w, 4), dtype=torch.float32, device="cuda")
    elif case["entry"] in ("render", "load"):
        s["out"] = np.zeros((h, w, 4), np.float32)
    return s


def run(s):
    case, ctx, entry = s["case"], s["ctx"], s["case"]["entry"]
    kw = {"samples": case["spp"], "sample_offset": s["offset"], "max_depth": case["depth"]}
    if entry == "batch":
        return ctx.render_batch(s["jobs"], case["algo"])[0]
    if entry == "f64":
        return ctx.render_f64(case["w"], case["h"], **kw)
    if entry == "device":
        ctx.render_device(s["out"].data_ptr(), case["w"], case["h"], **kw)
        return s["out"]
    if entry == "noalloc":
        ctx.render_noalloc(s["out"].data_ptr(), case["w"], case["h"], **kw)
        return s["out"]
    if entry == "load":
        ctx.load_scene_arrays(s["arrays"])
        ctx.set_camera(*s["cam"])
    return ctx.render(case["w"], case["h"], out=s["out"], **kw)[0]


def work(case):
    """What a pass cannot do without.  Bytes: each triangle's vertices and the
    picture, once.  Operations: for each path segment one descent of a binary
    tree over the triangles (two box tests of 18 operations a level), one
    triangle test (45) and its shading (150); a load adds 60 a triangle."""
    tris = case["tris"]
    pixels, samples, n = case["w"] * case["h"], case["w"] * case["h"] * case["spp"], 1
    if case["entry"] == "batch":
        n = case["jobs"]
        samples = sum(case["w"] * case["h"] * max(1, case["spp"] >> (k % 3)) for k in range(n))
    per_segment = 36 * max(1.0, math.log2(max(2, tris))) + 45 + 150
    segments = min(SEGMENTS[case["scene"]], case["depth"])
    load = 60 * tris if case["entry"] == "load" else 0
    return {"bytes": 36 * tris * n + pixels * n * (32 if case["entry"] == "f64" else 16),
            "flops": samples * segments * per_segment + load}


def exact(case, seed):
    """None: a path is a chain of decisions on single-precision values, so a
    64-bit evaluation of the same seed follows other paths."""
    return None
