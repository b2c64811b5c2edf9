"""GPU tests of the device BVH build at the sizes where its steps can go wrong:
the smallest trees, odd sizes, coincident and degenerate triangles, one long
chain of boxes.  Every sample's primary hit, event hash and shadow counts
equal the CPU oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _triangles(kind, n):
    rng = np.random.default_rng(n)
    if kind == "random":
        c = rng.uniform(-1.0, 1.0, (n, 1, 3))
        v = c + rng.uniform(-0.15, 0.15, (n, 3, 3))
    elif kind == "coincident":   # groups of equal triangles: equal Morton codes and boxes
        c = rng.uniform(-1.0, 1.0, (max(1, n // 7), 1, 3))
        v = (c + rng.uniform(-0.3, 0.3, (max(1, n // 7), 3, 3)))[np.arange(n) % max(1, n // 7)]
    elif kind == "long":         # every one spans the scene: more than the list of large ones holds
        a = rng.uniform(-1.0, 1.0, (n, 1, 3))
        v = np.concatenate([a, -a, a + rng.uniform(-0.02, 0.02, (n, 1, 3))], 1)
    elif kind == "degenerate":   # points and slivers among the others
        v = rng.uniform(-1.0, 1.0, (n, 1, 3)) + rng.uniform(-0.2, 0.2, (n, 3, 3))
        v[::3, 1] = v[::3, 0]
        v[::5, 2] = v[::5, 0]
    else:                        # a chain along x, sizes growing along it
        s = 0.002 * 1.004 ** np.arange(n)
        x = np.cumsum(s) / max(1e-9, s.sum()) * 2.0 - 1.0
        v = np.stack([np.stack([x, 0 * x, 0 * x], 1), np.stack([x + s, 0 * x, 0.1 + 0 * x], 1),
                      np.stack([x, 0.3 + 0 * x, 0.05 + 0 * x], 1)], 1)
    return v.astype(np.float32).reshape(-1, 3).astype(np.float64), np.arange(3 * n).reshape(n, 3)


@pytest.mark.parametrize("kind,n", [("random", 1), ("random", 4), ("random", 5), ("random", 6), ("random", 9),
                                    ("random", 33), ("random", 257), ("random", 4097), ("coincident", 5),
                                    ("coincident", 700), ("degenerate", 300), ("chain", 900), ("long", 40),
                                    ("long", 4100)])
def test_small_and_awkward_trees_match_the_oracle(kind, n):
    import lucid_capi
    import lucid_scenes as ls
    from parity_util import render_gpu, render_oracle
    v, t = _triangles(kind, n)
    light = {"type": "POINT", "position": [1.5, 2.0, 2.5], "color": [1, 1, 1], "energy": 200.0, "radius": 0.0}
    scene = {"meshes": [ls.mesh(v, t, ls.material((0.6, 0.5, 0.4), 0.0, 0.6))], "native_lights": [light],
             "environment": {"color": [0.2, 0.2, 0.3], "strength": 1.0}}
    cam = (0.1, 0.15, 3.1, 0.0, -0.02, -1.0, 0.0, 1.0, 0.0, 50.0)
    ctx = lucid_capi.Context(0)
    img, recs = render_gpu(ctx, scene, cam, "mis", 40, 36, 2, 4)
    ctx.close()
    ref, rref = render_oracle(scene, cam, "mis", 40, 36, 2, 4)
    assert n < 5 or (rref["primary_mesh"] >= 0).any()
    for f in ("primary_mesh", "primary_tri", "bounces", "nee_tests", "nee_occluded", "hash"):
        np.testing.assert_array_equal(recs[f], rref[f])
    np.testing.assert_allclose(img, ref, rtol=1e-4, atol=1e-5)


def test_a_context_reloads_scenes_of_other_sizes():
    """One context through scenes that grow and shrink, with and without
    lights, media and large triangles: each renders as on a context of its
    own."""
    import lucid_capi
    import lucid_scenes as ls
    from parity_util import render_gpu
    room, rcam = ls.cornell_variant(3, 5000)
    v, t = _triangles("random", 60)
    few = {"meshes": [ls.mesh(v, t, ls.material((0.6, 0.5, 0.4), 0.0, 0.6))], "native_lights": [],
           "environment": {"color": [0.2, 0.2, 0.3], "strength": 1.0}}
    fcam = (0.1, 0.15, 3.1, 0.0, -0.02, -1.0, 0.0, 1.0, 0.0, 50.0)
    lit, lcam = ls.all_lights_scene("/tmp")
    order = [(room, rcam), (few, fcam), (lit, lcam), (few, fcam), (room, rcam), (lit, lcam)]
    one = lucid_capi.Context(0)
    for scene, cam in order:
        got, grec = render_gpu(one, scene, cam, "volume_mis", 48, 40, 2, 6)
        own = lucid_capi.Context(0)
        want, wrec = render_gpu(own, scene, cam, "volume_mis", 48, 40, 2, 6)
        own.close()
        np.testing.assert_array_equal(got, want)
        np.testing.assert_array_equal(grec, wrec)
    one.close()
