"""The depth stage's tile culling against the per-fragment restatement, bit for bit: every tile
size, images that no tile size divides, sprites cut by the image and by the near plane, sprites
of more than 32 tiles, ties, and a view whose sprites are too small for tiles."""
import numpy as np
import pytest
import torch

from fluids_gb300 import capi, render
from oracle import render as orender

pytestmark = pytest.mark.gpu


def _particles(n, seed):
    """A dense block seen from a corner, a sheet near the camera, strays in and out of view."""
    rng = np.random.default_rng(seed)
    p = np.ones((n, 4), np.float32)
    a, b = n // 2, n // 4
    p[:a, :3] = rng.uniform(-0.4, 0.4, (a, 3))
    p[a:a + b, :3] = rng.uniform(-0.3, 0.3, (b, 3)) * (1, 0.02, 1) + (0, 0.9, 0.9)
    p[a + b:, :3] = rng.uniform(-3.0, 3.0, (n - a - b, 3))
    p[1::50] = p[0]   # ties: the lowest index wins
    return p


@pytest.mark.parametrize("w,h,size", [(97, 61, 7.0), (130, 113, 13.0), (161, 95, 30.0), (203, 149, 70.0),
                                      (64, 64, 12.0), (97, 61, 3.0)])
def test_depth_with_tiles_matches_restatement(gpu_lib, w, h, size):
    p = _particles(3000, int(size))
    cam = render.Camera(w, h)
    mv, pr = cam.transformation(), cam.projection()
    radius = size * 4.0 / cam.point_scale()   # that many pixels at the scene's origin
    ctx = capi.Context(capi.make_params(capi.SPH_WCSPH, mode=capi.SPH_MODE_PHYSICS))
    ctx.set_rect_limits(8.0, 8.0, 8.0)
    ctx.add_volume(p)
    depth = torch.zeros((h, w), dtype=torch.float32, device="cuda")
    ctx.render_depth(capi.make_view(mv, pr, radius, cam.point_scale(), w, h), depth.data_ptr())
    ctx.synchronize()
    want = orender.splat_depth(p, mv, pr, radius, cam.point_scale(), w, h)
    assert np.array_equal(depth.cpu().numpy(), want)
    assert (want > 0).any()


def test_bilateral_edges_match_restatement(gpu_lib):
    """Images smaller than a block, wider by one pixel, and with empty blocks."""
    for w, h in ((1, 1), (31, 9), (33, 8), (70, 41)):
        rng = np.random.default_rng(w)
        d = rng.uniform(0.8, 0.81, (h, w)).astype(np.float32)
        d[rng.uniform(size=(h, w)) < 0.3] = 0.0
        d[:, w // 2:] *= (w < 60)
        a, b = torch.from_numpy(d).cuda(), torch.zeros((h, w), device="cuda")
        capi.filter_bilateral(a.data_ptr(), b.data_ptr(), w, h)
        torch.cuda.synchronize()
        # expf's last place in 64 weights of about 1, as the golden comparison has it
        np.testing.assert_allclose(b.cpu().numpy(), orender.bilateral(d), rtol=0, atol=2e-6)
