"""GPU test of the film sum that writes the picture of a call whose samples are
one wave: each pixel is the sum of its samples' radiance in sample order, bit
for bit, for sample counts around its load groups (of 8)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,spp", [(7, 5, 1), (7, 5, 2), (1, 1, 7), (5, 3, 8), (1, 3, 9), (13, 11, 15), (13, 11, 16),
                                     (13, 11, 17), (3, 1, 24), (1, 1, 4099), (129, 1, 31)])
def test_picture_is_the_ordered_sum_of_its_samples(w, h, spp):
    import lucid_capi
    import lucid_scenes as ls
    sc, cam = ls.cornell_box()
    ctx = lucid_capi.Context(0)
    try:
        ctx.load_scene_json(ls.to_json(sc))
        ctx.set_camera(*cam)
        ctx.set_algorithm("mis")
        img, recs, _ = ctx.render(w, h, samples=spp, sample_offset=3, records=True)
        rgb = recs["rgb"].reshape(h, w, spp, 3)
        want = np.zeros((h, w, 3), np.float32)
        for s in range(spp):
            want = want + rgb[:, :, s]
        np.testing.assert_array_equal(img[..., :3], np.maximum(want, np.float32(0))[::-1])
        assert (img[..., 3] == 1).all()
    finally:
        ctx.close()
