"""The PCISPH loop in one launch, its predictions and integration as epilogues of the force
pass, against its passes one by one: at sizes on both sides of one and of three rounds of five
blocks an SM (152 SMs), beyond which a denser variant runs."""
import numpy as np
import pytest

from fluids_gb300 import capi
from fluids_gb300.scenes import FishTank, jitter, lattice_block

pytestmark = pytest.mark.gpu

DX, BOX, ITERS = 0.008, (1.0, 0.9, 0.9), 4
SETUP = ("BOUNDARY_SYNC", "HASHES", "SORT", "SHUFFLE", "CELL_INTERVALS", "NEIGH_LIST", "PCI_INIT_DENSITY", "NORMALS",
         "PCI_INIT_FORCES")


def _context(n):
    k = int(np.ceil(n ** (1.0 / 3.0)))
    p = jitter(lattice_block(k, k, k, DX, (-0.5 + DX, -0.45 + DX, -0.45 + DX)), 2e-4, n)[:n]
    ctx = capi.Context(capi.make_params(
        capi.SPH_PCISPH, mode=capi.SPH_MODE_PHYSICS, time_step=5e-5, particle_radius=DX / 2, support_radius=2 * DX,
        k_viscosity=1.7, gas_stiffness=2000.0, surface_tension=1.0, gravity=9.81, max_vel=20.0, relax_on_add=0,
        pcisph_min_iterations=ITERS, pcisph_max_iterations=ITERS))
    ctx.set_rect_limits(*BOX)
    ctx.add_boundary(FishTank(*BOX).surface_sampling(DX))
    ctx.add_volume(p, np.zeros_like(p))
    return ctx


@pytest.mark.parametrize("n", [1, 2049, 194560, 194561, 583680, 583681])
def test_loop_equals_its_passes(gpu_lib, n):
    a, b, whole = _context(n), _context(n), _context(n)
    for s in SETUP:
        a.stage(s)
        b.stage(s)
    a.stage("PCI_LOOP")
    for _ in range(ITERS):
        for s in ("PCI_PREDICT", "PCI_UPDATE_PRESSURE", "PCI_PRESSURE_FORCE"):
            b.stage(s)
    assert a.get("PCI_ITERS")[0] == ITERS
    # the passes' arithmetic is the loop's; where the compiler contracts an expression of the two
    # differently, a last bit of a predicted position (6e-8 of a support radius of 1.6e-2) changes
    # a density of 1000 by up to 1e-2 against errors of tens: 1e-3
    for f, rtol in (("POS_PRED", 1e-6), ("PRESSURE", 1e-3), ("FORCE_PRESSURE", 1e-3)):
        x, y = (c.get(f).astype(np.float64) for c in (a, b))
        assert np.abs(x - y).max() <= rtol * max(np.abs(y).max(), 1e-30), f
    whole.simulate(1)
    b.stage("PCI_INTEGRATE")
    assert np.array_equal(whole.get("ID"), b.get("ID"))
    # one step moves a particle by dt^2 times its acceleration: far below the bound's 1e-6
    x, y = (c.get("POS").reshape(-1, 4)[:, :3].astype(np.float64) for c in (whole, b))
    assert np.abs(x - y).max() <= 1e-6 * np.abs(y).max()
    x, y = (c.get("VEL").reshape(-1, 4)[:, :3].astype(np.float64) for c in (whole, b))
    assert np.abs(x - y).max() <= 1e-3 * max(np.abs(y).max(), 1e-30)
