"""A PCISPH step with a particle that is not a number: it has no neighbours, so its normal and its
pressure force are zero, with one lane a particle and with several, and no other particle sees it."""
import numpy as np
import pytest

from fluids_gb300 import capi
from fluids_gb300.scenes import FishTank, jitter, lattice_block

pytestmark = pytest.mark.gpu

DX, BOX = 0.012, (1.0, 0.9, 0.9)


@pytest.mark.parametrize("side", [3, 13, 23, 40])   # 8 lanes a particle up to 9,728, 4 up to 38,912, then 1
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_particle_that_is_not_a_number(gpu_lib, side, bad):
    ctx = capi.Context(capi.make_params(
        capi.SPH_PCISPH, mode=capi.SPH_MODE_PHYSICS, time_step=1e-4, particle_radius=DX / 2, support_radius=2 * DX,
        k_viscosity=1.7, gas_stiffness=2000.0, surface_tension=1.0, gravity=9.81, max_vel=20.0, relax_on_add=0,
        pcisph_min_iterations=3, pcisph_max_iterations=3))
    ctx.set_rect_limits(*BOX)
    ctx.add_boundary(FishTank(*BOX).surface_sampling(DX))
    ctx.add_volume(jitter(lattice_block(side, side, side, DX, (-0.4, -0.4, -0.3)), 3e-4, 1))
    for which in (5, side ** 3 - 1):
        pos = ctx.get("POS").reshape(-1, 4)
        pos[ctx.get("ID") == which, :3] = bad
        ctx.set("POS", pos)
    ctx.simulate(1)
    bad_ones = np.isin(ctx.get("ID"), (5, side ** 3 - 1))
    for f in ("NORMAL", "FORCE_PRESSURE"):
        x = ctx.get(f).reshape(-1, 4)[:, :3]
        assert not x[bad_ones].any() and np.isfinite(x).all(), f
    assert np.isfinite(ctx.get("POS").reshape(-1, 4)[~bad_ones]).all()
    assert ctx.device_flags() & capi.FLAGS["NAN"]
