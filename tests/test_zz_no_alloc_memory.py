"""GPU test that lucid_cuda_render_noalloc allocates no device memory, a process's
first call included: with almost none left it renders, and leaves as much."""
import os
import subprocess
import sys

import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu

CHILD = """
import sys
sys.path.insert(0, %r)
import torch
import lucid_capi
import lucid_scenes as ls
scene, cam = ls.cornell_box()
ctx = lucid_capi.Context(0)
ctx.load_scene_json(ls.to_json(scene))
ctx.set_camera(*cam)
ctx.set_algorithm(sys.argv[1])
out = torch.zeros((64, 64, 4), device="cuda")
torch.cuda.synchronize()
fill = torch.empty(torch.cuda.mem_get_info()[0] - (12 << 20), dtype=torch.uint8, device="cuda")
before = torch.cuda.mem_get_info()[0]
assert before < 16 << 20
ctx.render_noalloc(out.data_ptr(), 64, 64, 2, 0, 8)
assert torch.cuda.mem_get_info()[0] == before
assert float(out[..., :3].sum()) > 0
"""


@pytest.mark.parametrize("algo", ["simple", "nee", "mis", "volume_simple", "volume_mis"])
def test_first_call_of_a_process_allocates_nothing(algo):
    # a process of its own: in this one earlier tests have run the kernels
    r = subprocess.run([sys.executable, "-c", CHILD % PKG, algo], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ))
    assert r.returncode == 0, r.stderr[-1500:]
