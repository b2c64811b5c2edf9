"""GPU test of lucid_cuda_render_noalloc from several threads at once: every
context shares the device's one scratch array, and each call's image is still
its own.  Collected last, after test_zz_no_alloc.py."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_calls_of_several_contexts_keep_their_images():
    import torch
    import lucid_capi
    import lucid_scenes as ls
    jobs = []
    for k, (scene, algo, w, h, spp) in enumerate([(ls.cornell_box(), "mis", 96, 64, 4), (ls.material_preview_scene(2), "nee", 128, 128, 8),
                                                  (ls.cornell_variant(5, 2000), "simple", 61, 77, 30)]):
        ctx = lucid_capi.Context(0)
        ctx.load_scene_json(ls.to_json(scene[0]))
        ctx.set_camera(*scene[1])
        ctx.set_algorithm(algo)
        want = torch.zeros((h, w, 4), dtype=torch.float32, device="cuda")
        ctx.render_device(want.data_ptr(), w, h, spp, k, 8)
        jobs.append((ctx, w, h, spp, k, want.cpu().numpy(), torch.zeros((h, w, 4), dtype=torch.float32, device="cuda")))
    torch.cuda.synchronize()
    start = threading.Barrier(len(jobs))
    wrong = []

    def work(ctx, w, h, spp, offset, want, out):
        start.wait()
        for call in range(40):
            ctx.render_noalloc(out.data_ptr(), w, h, spp, offset, 8)
            got = out.cpu().numpy()
            if not np.array_equal(got, want):
                wrong.append((offset, call))
                return

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for j in jobs:
        j[0].close()
    assert not wrong
