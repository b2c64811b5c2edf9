"""GPU tests of the wavefront kernels, which only waves of more than 2^17 paths
reach: both launch profiles, the awkward trees at several depths, the camera
rays from inside the scene's coordinate bound, and scenes that are replaced
while another context renders them."""
import threading

import numpy as np
import pytest

from parity_util import scene_and_camera
from test_bvh_build import _triangles

pytestmark = pytest.mark.gpu

LINE = 1 << 17


def _context(scene, cam, algo):
    import lucid_capi
    import lucid_scenes as ls
    ctx = lucid_capi.Context(0)
    ctx.load_scene_json(ls.to_json(scene))
    ctx.set_camera(*cam)
    ctx.set_algorithm(algo)
    return ctx


@pytest.mark.parametrize("scene,algo,spp,depth", [("cornell", "mis", 112, 8), ("all_lights", "volume_mis", 112, 8),
                                                  ("procedural_small", "nee", 112, 6), ("two_volumes", "simple", 500, 5)])
def test_launch_profiles_give_identical_samples_in_large_waves(workdir, scene, algo, spp, depth):
    sc, cam = scene_and_camera(scene, workdir)
    ctx = _context(sc, cam, algo)
    try:
        w, h = 40, 30
        assert w * h * spp > LINE
        out = []
        for profile in (0, 1):
            ctx.set_launch_profile(profile)
            img, recs, _ = ctx.render(w, h, samples=spp, sample_offset=2, max_depth=depth, records=True)
            out.append((img, recs))
        np.testing.assert_array_equal(out[0][1], out[1][1])
        np.testing.assert_array_equal(out[0][0].view(np.uint32), out[1][0].view(np.uint32))
    finally:
        ctx.close()


@pytest.mark.parametrize("kind,n", [("random", 1), ("random", 4), ("random", 5), ("random", 33), ("random", 4097),
                                    ("coincident", 700), ("degenerate", 300), ("chain", 900), ("long", 40), ("long", 4100)])
def test_trees_in_large_waves_equal_the_whole_path_kernel(kind, n):
    """Bounces and shadow rays through the persistent traversal kernels: the
    single leaf, equal boxes, points and slivers, deep and overlapping trees."""
    import lucid_scenes as ls
    v, t = _triangles(kind, n)
    light = {"type": "POINT", "position": [1.5, 2.0, 2.5], "color": [1, 1, 1], "energy": 200.0, "radius": 0.0}
    scene = {"meshes": [ls.mesh(v, t, ls.material((0.6, 0.5, 0.4), 0.0, 0.6))], "native_lights": [light],
             "environment": {"color": [0.2, 0.2, 0.3], "strength": 1.0}}
    w, h = 40, 36
    spp = LINE // (w * h) + 1
    half = spp // 2
    ctx = _context(scene, (0.1, 0.15, 3.1, 0.0, -0.02, -1.0, 0.0, 1.0, 0.0, 50.0), "mis")
    try:
        _, recs, _ = ctx.render(w, h, samples=spp, max_depth=4, records=True)
        recs = recs.reshape(h, w, spp)
        assert n < 33 or ((recs["bounces"] > 1).any() and (recs["nee_tests"] > 0).any())
        for lo, hi in ((0, half), (half, spp)):
            _, r, _ = ctx.render(w, h, samples=hi - lo, sample_offset=lo, max_depth=4, records=True)
            np.testing.assert_array_equal(r.reshape(h, w, hi - lo), recs[:, :, lo:hi])
    finally:
        ctx.close()


@pytest.mark.parametrize("inside", [True, False])
@pytest.mark.parametrize("kind,n,w,h", [("random", 4, 37, 29), ("random", 5, 1, 1), ("random", 4097, 33, 31),
                                        ("coincident", 700, 9, 4), ("degenerate", 300, 64, 32), ("chain", 900, 40, 5),
                                        ("long", 4100, 24, 24)])
def test_camera_walk_on_either_side_of_the_coordinate_bound(kind, n, w, h, inside):
    """The camera kernel in its FMA form (the camera's coordinates within the
    scene's largest) and in the subtraction form, just beyond it."""
    import lucid_scenes as ls
    v, t = _triangles(kind, n)
    scene = {"meshes": [ls.mesh(v, t, ls.material((0.6, 0.5, 0.4), 0.0, 0.6))], "native_lights": [],
             "environment": {"color": [0.2, 0.2, 0.3], "strength": 1.0}}
    bound = float(np.abs(v.astype(np.float32)).max())
    z = bound * (0.97 if inside else 1.03)
    assert (z <= bound) == inside and bound > 0.1
    spp = LINE // (w * h) + 1
    half = spp // 2
    ctx = _context(scene, (0.05, 0.04, z, 0.0, -0.02, -1.0, 0.0, 1.0, 0.0, 70.0), "simple")
    try:
        _, recs, _ = ctx.render(w, h, samples=spp, max_depth=1, records=True)
        recs = recs.reshape(h, w, spp)
        for lo, hi in ((0, half), (half, spp)):
            _, r, _ = ctx.render(w, h, samples=hi - lo, sample_offset=lo, max_depth=1, records=True)
            np.testing.assert_array_equal(r.reshape(h, w, hi - lo), recs[:, :, lo:hi])
    finally:
        ctx.close()


def test_scenes_replaced_while_another_context_renders_them():
    """A context loads one scene after another while batches of a second context
    render whichever it holds: every image is one of the scenes', whole."""
    import lucid_capi
    import lucid_scenes as ls
    scenes = [ls.cornell_variant(3, 3000), ls.cornell_variant(4, 5000), ls.cornell_box()]
    texts = [ls.to_json(s) for s, _ in scenes]
    cam = scenes[0][1]
    owner, other = lucid_capi.Context(0), lucid_capi.Context(0)
    try:
        job = {"scene": owner, "camera": cam, "width": 80, "height": 60, "samples": 4}
        want = []
        for text in texts:
            owner.load_scene_json(text)
            want.append(other.render_batch([job], "mis")[0][0])
        assert not np.array_equal(want[0], want[1]) and not np.array_equal(want[1], want[2])
        done, seen, wrong = threading.Event(), set(), []

        def render():
            while not done.is_set():
                img = other.render_batch([job, job], "mis")[0]
                for i in img:
                    k = [n for n, w in enumerate(want) if np.array_equal(i, w)]
                    if not k:
                        wrong.append(i)
                        return
                    seen.add(k[0])

        t = threading.Thread(target=render)
        t.start()
        for k in range(60):
            owner.load_scene_json(texts[k % 3])
        done.set()
        t.join()
        assert not wrong and seen
    finally:
        owner.close()
        other.close()
