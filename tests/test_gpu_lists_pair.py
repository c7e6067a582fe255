"""The fused step's list pass with two threads a particle (mid-size scenes with walls) against
the stage path's one-thread list kernel, on both sides of its limits (60,800 and 116,736
particles on 152 SMs), for one scene and for a batch: lists, order and lengths equal, densities
within the rounding of their sums."""
import numpy as np
import pytest

from fluids_gb300 import capi, workloads
from fluids_gb300.scenes import FishTank

pytestmark = pytest.mark.gpu

DX, CAP = 0.02, 50


def _fluid(n, seed, box):
    """n particles, about eight a cell, from the floor's and two walls' cells up."""
    side = (n / 8.0) ** (1.0 / 3.0) * 2 * DX
    p = np.ones((n, 4), np.float32)
    p[:, :3] = np.random.default_rng(seed).uniform(0.0, side, (n, 3)) - np.array(box) / 2 + 0.3 * DX
    return p


def _single(n, method):
    box = (1.2, 1.1, 1.1)
    kw = dict(mode=capi.SPH_MODE_PHYSICS, time_step=1e-5, particle_radius=DX / 2, support_radius=2 * DX,
              surface_tension=0.001, gravity=9.81)
    if method == capi.SPH_PCISPH:
        kw.update(relax_on_add=0, pcisph_max_iterations=3)
    ctx = capi.Context(capi.make_params(method, **kw))
    ctx.set_rect_limits(*box)
    ctx.add_boundary(FishTank(*box).surface_sampling(DX))
    ctx.add_volume(_fluid(n, n, box))
    return ctx


def _batch(n, _):
    parts, boxes = [n // 3, 1, n - n // 3 - 1], [(0.9, 0.8, 0.8), (0.4, 0.4, 0.4), (1.1, 1.0, 1.0)]
    return capi.BatchContext(workloads.wcsph_params(DX, 1e-5), [
        dict(container=b, mu=0.01, kgas=1000.0, fluid=_fluid(m, m + k, b), boundary=FishTank(*b).surface_sampling(DX))
        for k, (m, b) in enumerate(zip(parts, boxes))])


@pytest.mark.parametrize("make,method", [(_single, capi.SPH_WCSPH), (_single, capi.SPH_PCISPH), (_batch, capi.SPH_WCSPH)])
@pytest.mark.parametrize("n", [60800, 60801, 116736, 116737])
def test_pair_lists_equal_stage_lists(gpu_lib, make, method, n):
    a, b = make(n, method), make(n, method)
    a.simulate(1)
    for s in ("BOUNDARY_SYNC", "HASHES", "SORT", "SHUFFLE", "CELL_INTERVALS", "NEIGH_LIST"):
        b.stage(s)
    b.stage("WC_DENSITY" if method == capi.SPH_WCSPH else "PCI_INIT_DENSITY")
    for kind in ("NEIGH", "SB_NEIGH"):
        la, lb = a.get(kind + "_LEN"), b.get(kind + "_LEN")
        assert np.array_equal(la, lb) and la.max() > 0
        ea, eb = a.get(kind + "_LIST").reshape(CAP, n), b.get(kind + "_LIST").reshape(CAP, n)
        used = np.arange(CAP)[:, None] < la[None, :]
        assert np.array_equal(ea[used], eb[used])
    # at most two sums of at most 2 cap positive terms, each rounded to 2^-24
    da, db = a.get("DENSITY"), b.get("DENSITY")
    assert np.all(np.abs(da - db) <= 2 * (2 * CAP + 8) * 2.0 ** -24 * np.abs(db))
