"""Batched steps: one tile per warp, or several lanes a particle in small batches, against the
stage path's one-thread walks; one step's state at batch sizes on both sides of every change
of the lane count, with scenes whose last tiles are partial."""
import numpy as np
import pytest

from fluids_gb300 import capi, workloads
from fluids_gb300.scenes import FishTank, jitter, lattice_block

pytestmark = pytest.mark.gpu

DX = 0.015


def _scenes(n):
    """Three scenes of uneven size (one of a single particle, where there are enough) with n
    particles in all, in containers of different grids."""
    parts = [n] if n < 3 else [1, (n - 1) // 3, n - 1 - (n - 1) // 3]
    got = []
    for k, m in enumerate(parts):
        box = (0.9 + 0.3 * k, 0.8 + 0.1 * k, 0.8)
        side = int(np.ceil(m ** (1.0 / 3.0)))
        p = jitter(lattice_block(side, side, side, DX, tuple(DX - b / 2 for b in box)), 2e-4, m + k)[:m]
        v = np.zeros_like(p)
        v[:, :3] = np.random.default_rng(m + k).uniform(-0.5, 0.5, (m, 3))
        got.append(dict(container=box, mu=0.01 * (k + 1), kgas=1000.0 + 500.0 * k, fluid=p, vel=v,
                        boundary=FishTank(*box).surface_sampling(DX)))
    return got


# 8 | 4 | 2 | 1 lanes on 152 SMs (19,456, 38,912, 77,824)
@pytest.mark.parametrize("n", [1, 33, 2049, 19456, 19457, 38912, 38913, 77824, 77825])
@pytest.mark.parametrize("sigma", [0.001, 0.0])
def test_batched_step_equals_one_thread_walks(gpu_lib, n, sigma):
    p = workloads.wcsph_params(DX, 5e-5)
    p.surface_tension = sigma
    a, b = (capi.BatchContext(p, _scenes(n)) for _ in range(2))
    a.simulate(1)
    for s in ("BOUNDARY_SYNC", "HASHES", "SORT", "SHUFFLE", "CELL_INTERVALS", "NEIGH_LIST", "WC_DENSITY", "NORMALS",
              "WC_ACCEL", "WC_INTEGRATE"):
        if s != "NORMALS" or sigma != 0.0:
            b.stage(s)
    assert np.array_equal(a.get("ID"), b.get("ID"))
    assert np.array_equal(a.get("NEIGH_LEN"), b.get("NEIGH_LEN"))
    # sums of at most 50 terms in another order, and the packed records' reciprocals: the parity
    # bar of the float fields, 1e-5 of the largest value
    for f, rtol in [("POS", 1e-6), ("VEL", 1e-5)] + ([("NORMAL", 1e-5)] if sigma else []):
        x, y = (c.get(f).reshape(-1, 4)[:, :3].astype(np.float64) for c in (a, b))
        assert np.abs(x - y).max() <= rtol * max(np.abs(y).max(), 1e-30)
