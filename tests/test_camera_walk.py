"""GPU test of the camera rays' walk over the binary tree (its leaf-to-leaf
loop, the entries it drops and the interruption for few walking lanes): waves
large enough for the camera-ray kernel give the same records and image as the
same samples in waves small enough for the whole-path kernel, whose traversal
is another one; from inside the scene's coordinate bound and from outside it."""
import numpy as np
import pytest

from test_bvh_build import _triangles

pytestmark = pytest.mark.gpu

LINE = 1 << 17   # paths up to which a wave is the whole-path kernel's


@pytest.mark.parametrize("far", [False, True])
@pytest.mark.parametrize("kind,n,w,h", [("random", 4, 37, 29),       # one leaf
                                        ("random", 5, 1, 1),         # one lane a warp
                                        ("random", 4097, 33, 31),    # ragged tiles
                                        ("coincident", 700, 9, 4),   # equal distances
                                        ("degenerate", 300, 64, 32),
                                        ("chain", 900, 40, 5),       # deep tree
                                        ("long", 4100, 24, 24)])     # overlapping boxes
def test_camera_kernel_equals_the_whole_path_kernel(kind, n, w, h, far):
    import lucid_capi
    import lucid_scenes as ls
    v, t = _triangles(kind, n)
    scene = {"meshes": [ls.mesh(v, t, ls.material((0.6, 0.5, 0.4), 0.0, 0.6))], "native_lights": [],
             "environment": {"color": [0.2, 0.2, 0.3], "strength": 1.0}}
    z, fov = (60.0, 3.0) if far else (1.1, 60.0)
    spp = LINE // (w * h) + 1
    half = spp // 2
    ctx = lucid_capi.Context(0)
    try:
        ctx.load_scene_json(ls.to_json(scene))
        ctx.set_camera(0.1, 0.05, z, 0.0, -0.02, -1.0, 0.0, 1.0, 0.0, fov)
        ctx.set_algorithm("simple")
        _, recs, _ = ctx.render(w, h, samples=spp, max_depth=1, records=True)
        recs = recs.reshape(h, w, spp)
        for lo, hi in ((0, half), (half, spp)):
            _, r, _ = ctx.render(w, h, samples=hi - lo, sample_offset=lo, max_depth=1, records=True)
            np.testing.assert_array_equal(r.reshape(h, w, hi - lo), recs[:, :, lo:hi])
    finally:
        ctx.close()
