"""The scratch that the particle renderer keeps: 8 bytes a pixel, the order's 16 a particle and its
sort's workspace, and not the depth stage's list of pairs."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import numpy as np, torch
from fluids_gb300 import capi, render
n, w, h = 2_000_000, 64, 48
p = np.ones((n, 4), np.float32)
p[:, :3] = np.random.default_rng(1).uniform(-0.9, 0.9, (n, 3))
ctx = capi.Context(capi.make_params(capi.SPH_WCSPH, mode=capi.SPH_MODE_PHYSICS, relax_on_add=0))
ctx.set_rect_limits(2.0, 2.0, 2.0)
ctx.add_volume(p)
rgba = torch.zeros((h, w, 4), device="cuda")
cam = render.Camera(w, h)
view = capi.make_view(cam.transformation(), cam.projection(), 0.0625, cam.point_scale(), w, h)
capi.sort_pairs_device(torch.zeros(8, dtype=torch.int32, device="cuda").data_ptr(),
                       torch.zeros(8, dtype=torch.int32, device="cuda").data_ptr(), 8)
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
ctx.render_particles(view, [((0.0, -1.0, 0.0), (1.0, 1.0, 1.0, 1.0))], rgba.data_ptr())
ctx.synchronize()
used = free - torch.cuda.mem_get_info()[0]
assert used <= 16 * n + 2 * 256 * 4 * (n // 4096 + 1) + (8 << 20), used
print("held", used)
"""


def test_particles_hold_no_pair_list(gpu_lib):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CODE], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "held" in r.stdout, r.stdout + r.stderr
