"""GPU test: a diagnostic render gives back what it creates for one call."""
import pytest

pytestmark = pytest.mark.gpu


def _rss_kb():
    with open("/proc/self/statm") as f:
        return int(f.read().split()[1]) * 4


def test_diagnostic_renders_do_not_grow_the_process():
    import lucid_capi
    import lucid_scenes as ls
    sc, cam = ls.cornell_box()
    ctx = lucid_capi.Context(0)
    try:
        ctx.load_scene_json(ls.to_json(sc))
        ctx.set_camera(*cam)
        ctx.set_algorithm("mis")
        ctx.diag_enable()
        for _ in range(500):
            ctx.render(8, 8, samples=1)
        before = _rss_kb()
        for _ in range(4000):
            ctx.render(8, 8, samples=1)
        # two CUDA events kept a call are 1.2 KB: 4.8 MB here
        assert _rss_kb() - before < 1024
    finally:
        ctx.close()
