"""GPU tests of rays with direction components that are exactly 0, against the
CPU oracle: shadow rays to a sun straight overhead of a tessellated object that
stands on both sides of the coordinate planes, and the centre column and row of
an unjittered camera along an axis; in waves of the whole-path kernel (up to
2^17 paths) and of the wavefront kernels (above), and in a batch."""
import numpy as np
import pytest

from parity_util import compare_records, render_gpu, render_oracle

pytestmark = pytest.mark.gpu

LINE = 1 << 17


def _scene(sun, volume=None):
    import lucid_scenes as ls
    v, t = ls.icosphere(4)   # 5,120 triangles around the origin
    meshes = [ls.mesh(v * 0.7, t, ls.material((0.7, 0.4, 0.3), 0.0, 0.8)),
              ls.mesh(*ls.quad((-4, -1.1, -4), (-4, -1.1, 4), (4, -1.1, 4), (4, -1.1, -4)), ls.material((0.5, 0.5, 0.5), 0.0, 1.0)),
              ls.mesh(*ls.quad((-3, -1.1, -3), (-3, 3, -3), (-3, 3, 3), (-3, -1.1, 3)), ls.material((0.4, 0.5, 0.6), 0.0, 1.0))]
    if volume:
        meshes.append(ls.volume_box_mesh((-0.9, -0.9, -0.9), (0.9, 0.9, 0.9), 0.4, (0.9, 0.8, 0.7), 0.1, volume, (4, 4, 4)))
    return {"meshes": meshes, "native_lights": [{"type": "SUN", "direction": sun, "color": [1, 1, 1], "energy": 3.0}],
            "environment": {"color": [0.2, 0.25, 0.3], "strength": 1.0}}


SUNS = {"y": [0.0, -1.0, 0.0], "x": [-1.0, 0.0, 0.0], "yz": [0.0, -0.8, -0.6]}   # "x": the shadow is on the wall
OBLIQUE = (0.3, 1.2, 3.5, -0.02, -0.35, -1.0, 0.0, 1.0, 0.0, 50.0)
ALONG_Z = (0.2, 0.15, 3.0, 0.0, 0.0, -1.0, 0.0, 1.0, 0.0, 50.0)


def _same(scene, cam, algo, w, h, spp, depth):
    import lucid_capi
    ctx = lucid_capi.Context(0)
    try:
        img, recs = render_gpu(ctx, scene, cam, algo, w, h, spp, depth)
        ref, rref = render_oracle(scene, cam, algo, w, h, spp, depth)
        r = compare_records(recs, rref)
        assert r["primary"] == 0 and r["hash"] == 0 and r["counts"] == 0 and r["rgb"] == 0, r
        np.testing.assert_allclose(img, ref, rtol=1e-4, atol=1e-5)
        return ctx, img, rref
    except BaseException:
        ctx.close()
        raise


@pytest.mark.parametrize("w,h", [(97, 61), (401, 333)])   # below and above the line
@pytest.mark.parametrize("sun,algo", [("y", "nee"), ("x", "nee"), ("yz", "mis"), ("y", "volume_mis")])
def test_sun_along_an_axis_casts_the_oracles_shadow(tmp_path, sun, algo, w, h):
    import lucid_scenes as ls
    grid = None
    if algo == "volume_mis":
        grid = str(tmp_path / "grid.f32")
        ls.write_constant_grid(grid, (4, 4, 4), 1.0)
    ctx, _, rref = _same(_scene(SUNS[sun], grid), OBLIQUE, algo, w, h, 1, 4)
    ctx.close()
    assert (w * h > LINE) == (w > 100)
    assert (rref["nee_occluded"] > 0).any()


@pytest.mark.parametrize("w,h", [(97, 61), (401, 333)])
def test_unjittered_camera_along_an_axis(w, h):
    scene = _scene(SUNS["yz"])
    ctx, img, rref = _same(scene, ALONG_Z, "mis", w, h, 1, 3)
    try:
        column = rref["primary_mesh"].reshape(h, w)[:, w // 2]
        assert (column == 0).any() and (column == 1).any()   # the sphere and the ground
        batch, _ = ctx.render_batch([{"scene": ctx, "camera": ALONG_Z, "width": w, "height": h, "samples": 1,
                                      "max_depth": 3}], "mis")
        np.testing.assert_array_equal(batch[0], img)
    finally:
        ctx.close()
