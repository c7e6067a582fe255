"""The fused step's list pass at the sizes where it splits a particle over lanes, against the
stage path's one-thread list kernel: lists, order, cap and lengths equal, densities within the
rounding of their sums."""
import numpy as np
import pytest

from fluids_gb300 import capi
from fluids_gb300.scenes import FishTank

pytestmark = pytest.mark.gpu

DX, BOX = 0.02, (0.6, 0.5, 0.4)


def _fluid(n, crowd, seed):
    """n particles over a box of about n / crowd cells, some of them in the floor's cells."""
    rng = np.random.default_rng(seed)
    side = min(0.36, max(0.01, (n / crowd) ** (1.0 / 3.0) * 2 * DX))
    p = np.ones((n, 4), np.float32)
    p[:, :3] = rng.uniform(0.0, side, (n, 3)) + np.array([-0.28, -0.248, -0.19])
    return p


def _context(p, method, cap, block=0):
    kw = dict(mode=capi.SPH_MODE_PHYSICS, time_step=1e-5, particle_radius=DX / 2, support_radius=2 * DX,
              neigh_cap=cap, block_size=block, surface_tension=0.001, gravity=9.81)
    if method == capi.SPH_PCISPH:
        kw.update(relax_on_add=0, pcisph_max_iterations=3)
    ctx = capi.Context(capi.make_params(method, **kw))
    ctx.set_rect_limits(*BOX)
    ctx.add_boundary(FishTank(*BOX).surface_sampling(DX))
    ctx.add_volume(p)
    return ctx


# 8 lanes: a partial warp and block, cells of more than one and more than two rounds of a pair,
# full lists (cap 5 and 50), the longest cap the split pass takes and the next one
@pytest.mark.parametrize("method", [capi.SPH_WCSPH, capi.SPH_PCISPH])
@pytest.mark.parametrize("n,crowd,cap", [(1, 1, 50), (7, 1, 50), (33, 8, 50), (700, 8, 50), (700, 40, 50),
                                         (701, 12, 5), (1500, 20, 128), (1500, 20, 129)])
def test_split_lists_equal_stage_lists(gpu_lib, method, n, crowd, cap):
    p = _fluid(n, crowd, n + crowd)
    a, b = _context(p, method, cap), _context(p, method, cap)
    a.simulate(1)
    for s in ("BOUNDARY_SYNC", "HASHES", "SORT", "SHUFFLE", "CELL_INTERVALS", "NEIGH_LIST"):
        b.stage(s)
    b.stage("WC_DENSITY" if method == capi.SPH_WCSPH else "PCI_INIT_DENSITY")
    for kind in ("NEIGH", "SB_NEIGH"):
        la, lb = a.get(kind + "_LEN"), b.get(kind + "_LEN")
        assert np.array_equal(la, lb)
        ea, eb = a.get(kind + "_LIST").reshape(cap, n), b.get(kind + "_LIST").reshape(cap, n)
        used = np.arange(cap)[:, None] < la[None, :]
        assert np.array_equal(ea[used], eb[used])
    if crowd >= 20 and cap <= 50:
        assert a.get("NEIGH_LEN").max() == cap
    # at most two sums of at most 2 cap positive terms, each rounded to 2^-24
    da, db = a.get("DENSITY"), b.get("DENSITY")
    assert np.all(np.abs(da - db) <= 2 * (2 * cap + 8) * 2.0 ** -24 * np.abs(db))
