"""The depth stage where its work takes another way: sprites of very many tiles, a list of pairs
that is full, and large fluids whose sprites do or do not close the surface, each bit for bit
against the per-fragment restatement."""
import numpy as np
import pytest
import torch

from fluids_gb300 import capi, render
from oracle import render as orender

pytestmark = pytest.mark.gpu


def _depth(p, cam, radius, w, h, particle_radius=0.01):
    ctx = capi.Context(capi.make_params(capi.SPH_WCSPH, mode=capi.SPH_MODE_PHYSICS, particle_radius=particle_radius,
                                        support_radius=max(0.04, 2 * particle_radius)))
    ctx.set_rect_limits(8.0, 8.0, 8.0)
    ctx.add_volume(p)
    mv, pr, scale = cam.transformation(), cam.projection(), cam.point_scale()
    depth = torch.zeros((h, w), dtype=torch.float32, device="cuda")
    ctx.render_depth(capi.make_view(mv, pr, radius, scale, w, h), depth.data_ptr())
    ctx.synchronize()
    got = depth.cpu().numpy()
    ctx.close()
    want = orender.splat_depth(p, mv, pr, radius, scale, w, h)
    assert np.array_equal(got, want)
    return want


@pytest.mark.parametrize("zoom,radius", [(4.0, 0.9), (0.7, 0.2), (0.7, 0.02)])
def test_sprites_of_many_tiles(gpu_lib, zoom, radius):
    """Sprites of up to the whole image, and a camera among the particles, whose nearest sprites are
    many times as wide as those at the origin."""
    rng = np.random.default_rng(int(10 * zoom))
    p = np.ones((700, 4), np.float32)
    p[:, :3] = rng.uniform(-0.5, 0.5, (700, 3))
    p[1::40] = p[0]
    want = _depth(p, render.Camera(611, 407, zoom=zoom), radius, 611, 407)
    assert (want != 0).any()


def test_full_list_of_pairs(gpu_lib):
    """40,000 sprites side by side, whose tiles are more than the list's 2 n + 524,288 entries."""
    side, w = 200, 4096
    cam = render.Camera(w, w, roll=0.0)
    step = 19.0 / (0.5 * w / np.tan(np.radians(22.5)) / 4.0)   # 19 pixels at the camera's distance
    a = (np.arange(side) - 0.5 * (side - 1)) * step
    p = np.ones((side * side, 4), np.float32)
    p[:, 0], p[:, 1], p[:, 2] = np.tile(a, side), np.repeat(a, side), 0.0
    want = _depth(p, cam, 17.0 * 4.0 / cam.point_scale(), w, w)
    tiles = (want.reshape(w // 4, 4, w // 4, 4) != 0).any(axis=(1, 3)).sum()
    assert tiles > 2 * len(p) + 524_288   # at least one pair each


@pytest.mark.parametrize("particle_radius", [0.02, 0.15])
@pytest.mark.parametrize("n", [131_072, 131_073])
def test_open_and_closed_surfaces_of_large_fluids(gpu_lib, n, particle_radius):
    """Sprites of 9 pixels, 8.3 and 1.1 spacings wide, at the size from which the spacing counts;
    most particles lie outside the view."""
    rng = np.random.default_rng(n)
    p = np.ones((n, 4), np.float32)
    p[:, :3] = rng.uniform(-0.4, 0.4, (n, 3)) + (0.0, 0.0, 3.5)
    seen = rng.choice(n, 3000, replace=False)
    p[seen, :3] = rng.uniform(-0.4, 0.4, (3000, 3))
    cam = render.Camera(160, 90, roll=0.0)
    want = _depth(p, cam, 9.0 * 4.0 / cam.point_scale(), 160, 90, particle_radius)
    assert (want != 0).any()
