"""GPU tests of the split of a wave between the wavefront kernels and the
whole-path kernel (waves up to 2^17 paths, and the queues a larger wave leaves
at its end): the same samples rendered as one wave above the line and as tiles
below it give the same image and the same per-sample records bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LINE = 1 << 17


def _scene(name, tmp):
    import lucid_scenes as ls
    if name == "cornell":
        return ls.cornell_box()
    if name == "preview":
        return ls.material_preview_scene(4)
    if name == "textured":
        return ls.textured_scene()
    return ls.all_lights_scene(str(tmp))


def _context(name, algo, tmp):
    import lucid_capi
    import lucid_scenes as ls
    sc, cam = _scene(name, tmp)
    ctx = lucid_capi.Context(0)
    ctx.load_scene_json(ls.to_json(sc))
    ctx.set_camera(*cam)
    ctx.set_algorithm(algo)
    return ctx


@pytest.mark.parametrize("name,algo,w,h,spp,depth", [
    ("cornell", "mis", 363, 362, 1, 8),            # 131,406 paths: just above the line
    ("all_lights", "volume_mis", 211, 127, 5, 16),  # 133,985 paths, media and boundaries, long paths
    ("all_lights", "volume_simple", 333, 207, 2, 3),
    ("preview", "nee", 400, 333, 1, 2),
    ("textured", "simple", 640, 360, 3, 8),        # 691,200 paths: three wavefront depths
    ("cornell", "simple", 512, 512, 5, 1),         # one depth: no whole-path kernel
])
def test_wave_above_the_line_equals_tiles_below_it(tmp_path, name, algo, w, h, spp, depth):
    assert w * h * spp > LINE
    ctx = _context(name, algo, tmp_path)
    try:
        img, recs, _ = ctx.render(w, h, samples=spp, sample_offset=11, max_depth=depth, records=True)
        st = ctx.stats()
        recs = recs.reshape(h, w, spp)
        seg = shadow = 0
        rows = LINE // (w * spp) // 2
        for y in range(0, h, rows):
            n = min(rows, h - y)
            t, r, _ = ctx.render(w, n, w, h, samples=spp, sample_offset=11, max_depth=depth, tile_y=y, records=True)
            s = ctx.stats()
            seg += s["segments"]
            shadow += s["shadow_rays"]
            np.testing.assert_array_equal(t, img[h - y - n:h - y])
            np.testing.assert_array_equal(r.reshape(n, w, spp), recs[y:y + n])
        assert (seg, shadow) == (st["segments"], st["shadow_rays"])
    finally:
        ctx.close()


def test_device_and_batch_waves_agree_across_the_line(tmp_path):
    """One image on device memory, through the batch call alone and beside a
    second job that lifts the batch's wave above the line, and in waves cut to
    half its paths."""
    import torch
    w, h, spp = 200, 131, 4   # 104,800 paths
    ctx = _context("all_lights", "volume_mis", tmp_path)
    try:
        want, _, _ = ctx.render(w, h, samples=spp, max_depth=8)
        dev = torch.zeros((h, w, 4), dtype=torch.float32, device="cuda")
        ctx.render_device(dev.data_ptr(), w, h, samples=spp, max_depth=8)
        np.testing.assert_array_equal(dev.cpu().numpy(), want)
        import lucid_scenes as ls
        cam = ls.all_lights_scene(str(tmp_path))[1]
        job = {"scene": ctx, "camera": cam, "width": w, "height": h, "samples": spp}
        one, _ = ctx.render_batch([job], "volume_mis")
        two, _ = ctx.render_batch([job, dict(job, width=97, height=301)], "volume_mis")
        np.testing.assert_array_equal(one[0], want)
        np.testing.assert_array_equal(two[0], want)
        ctx.set_wave_capacity(w * h * 2)
        cut, _, _ = ctx.render(w, h, samples=spp, max_depth=8)
        np.testing.assert_array_equal(cut, want)
    finally:
        ctx.close()


def test_camera_far_outside_the_scene(tmp_path):
    """Whole paths whose camera rays take the subtraction slab form: the same
    picture as the wavefront's."""
    ctx = _context("cornell", "mis", tmp_path)
    try:
        ctx.set_camera(0.5, 0.5, 40.0, 0.0, 0.0, -1.0, 0.0, 1.0, 0.0, 2.0)
        big, _, _ = ctx.render(400, 400, samples=1, max_depth=8)
        small, _, _ = ctx.render(400, 200, 400, 400, samples=1, max_depth=8)
        assert float(big[..., :3].sum()) > 0
        np.testing.assert_array_equal(small, big[200:])
    finally:
        ctx.close()
