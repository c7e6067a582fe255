"""The PCISPH step with several lanes a particle and sums in list order, at the sizes where the
lane count changes (9,728 and 38,912 particles on 152 SMs): the loop against its one-thread
passes, and one whole step against the stage path."""
import numpy as np
import pytest

from fluids_gb300 import capi
from fluids_gb300.scenes import FishTank, jitter, lattice_block

pytestmark = pytest.mark.gpu

DX, BOX, ITERS = 0.012, (1.0, 0.9, 0.9), 4
SETUP = ("BOUNDARY_SYNC", "HASHES", "SORT", "SHUFFLE", "CELL_INTERVALS", "NEIGH_LIST", "PCI_INIT_DENSITY", "NORMALS",
         "PCI_INIT_FORCES")


def _context(n):
    k = int(np.ceil(n ** (1.0 / 3.0)))
    p = jitter(lattice_block(k, k, k, DX, (-0.5 + DX, -0.45 + DX, -0.45 + DX)), 3e-4, n)[:n]
    v = np.zeros_like(p)
    v[:, :3] = np.random.default_rng(n).uniform(-0.3, 0.3, (n, 3))
    ctx = capi.Context(capi.make_params(
        capi.SPH_PCISPH, mode=capi.SPH_MODE_PHYSICS, time_step=1e-4, particle_radius=DX / 2, support_radius=2 * DX,
        k_viscosity=1.7, gas_stiffness=2000.0, surface_tension=1.0, gravity=9.81, max_vel=20.0, relax_on_add=0,
        pcisph_min_iterations=ITERS, pcisph_max_iterations=ITERS))
    ctx.set_rect_limits(*BOX)
    ctx.add_boundary(FishTank(*BOX).surface_sampling(DX))
    ctx.add_volume(p, v)
    return ctx


@pytest.mark.parametrize("n", [1, 33, 9728, 9729, 38912, 38913])
def test_ordered_lanes_equal_one_thread_passes(gpu_lib, n):
    a, b, whole = _context(n), _context(n), _context(n)
    for s in SETUP:
        a.stage(s)
        b.stage(s)
    a.stage("PCI_LOOP")
    for _ in range(ITERS):
        for s in ("PCI_PREDICT", "PCI_UPDATE_PRESSURE", "PCI_PRESSURE_FORCE"):
            b.stage(s)
    # a last bit of a predicted position (6e-8 of a support radius of 2.4e-2) changes a density of
    # 1000 by up to 1e-2 against errors of tens: 1e-3
    for f, rtol in (("POS_PRED", 1e-6), ("PRESSURE", 1e-3), ("FORCE_PRESSURE", 1e-3)):
        x, y = (c.get(f).astype(np.float64) for c in (a, b))
        assert np.abs(x - y).max() <= rtol * max(np.abs(y).max(), 1e-30), f
    whole.simulate(1)
    b.stage("PCI_INTEGRATE")
    assert np.array_equal(whole.get("ID"), b.get("ID"))
    for f, rtol in (("NORMAL", 1e-5), ("FORCE_OTHER", 1e-5), ("POS", 1e-6), ("VEL", 1e-4)):
        x, y = (c.get(f).reshape(-1, 4)[:, :3].astype(np.float64) for c in (whole, b))
        assert np.abs(x - y).max() <= rtol * max(np.abs(y).max(), 1e-30), f
