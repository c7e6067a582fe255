"""The fused step's normal and force walks with several lanes a particle (small scenes),
against the stage path's one-thread walks: one step's state at sizes on both sides of every
change of the lane count."""
import numpy as np
import pytest

from fluids_gb300 import capi
from fluids_gb300.scenes import FishTank, jitter, lattice_block

pytestmark = pytest.mark.gpu

DX, BOX = 0.01, (1.0, 0.9, 0.9)
PCI = ("PCI_INIT_DENSITY", "NORMALS", "PCI_INIT_FORCES", "PCI_LOOP", "PCI_INTEGRATE")
WC = ("WC_DENSITY", "NORMALS", "WC_ACCEL", "WC_INTEGRATE")


def _context(n, method, sigma):
    k = int(np.ceil(n ** (1.0 / 3.0)))
    p = jitter(lattice_block(k, k, k, DX, (-0.5 + DX, -0.45 + DX, -0.45 + DX)), 2e-4, n)[:n]
    v = np.zeros_like(p)
    v[:, :3] = np.random.default_rng(n).uniform(-0.5, 0.5, (n, 3))
    kw = dict(mode=capi.SPH_MODE_PHYSICS, time_step=5e-5, particle_radius=DX / 2, support_radius=2 * DX,
              k_viscosity=0.05, gas_stiffness=2000.0, surface_tension=sigma, gravity=9.81, max_vel=20.0)
    if method == capi.SPH_PCISPH:
        kw.update(relax_on_add=0, pcisph_max_iterations=4, k_viscosity=1.7)
    ctx = capi.Context(capi.make_params(method, **kw))
    ctx.set_rect_limits(*BOX)
    ctx.add_boundary(FishTank(*BOX).surface_sampling(DX))
    ctx.add_volume(p, v)
    return ctx


# one particle; a partial warp and block; 8 | 4 | 2 | 1 lanes on 152 SMs (19,456, 38,912, 77,824)
@pytest.mark.parametrize("n", [1, 31, 2049, 19456, 19457, 38912, 38913, 77824, 77825])
@pytest.mark.parametrize("method,sigma", [(capi.SPH_WCSPH, 0.001), (capi.SPH_WCSPH, 0.0), (capi.SPH_PCISPH, 1.0)])
def test_lanes_equal_one_thread_walks(gpu_lib, n, method, sigma):
    a, b = _context(n, method, sigma), _context(n, method, sigma)
    a.simulate(1)
    for s in ("BOUNDARY_SYNC", "HASHES", "SORT", "SHUFFLE", "CELL_INTERVALS", "NEIGH_LIST"):
        b.stage(s)
    for s in WC if method == capi.SPH_WCSPH else PCI:
        if s != "NORMALS" or sigma != 0.0:
            b.stage(s)
    assert np.array_equal(a.get("ID"), b.get("ID"))
    # sums of at most 50 terms in another order, and the packed records' reciprocals: the parity
    # bar of the float fields, 1e-5 of the largest value (normals: each term is bounded by it
    # times the neighbour count)
    for f, rtol in [("POS", 1e-6), ("VEL", 1e-5)] + ([("NORMAL", 1e-5)] if sigma else []):
        x, y = (c.get(f).reshape(-1, 4)[:, :3].astype(np.float64) for c in (a, b))
        assert np.abs(x - y).max() <= rtol * max(np.abs(y).max(), 1e-30)
