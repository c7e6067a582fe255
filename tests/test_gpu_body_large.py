"""The forces on large bodies: the last size that takes several lanes a particle and the first that
takes a thread, and one whose forces run after the fluid's list pass instead of beside the rest
(152 SMs), by the stage and by the step, against the pair sum in float64."""
import numpy as np
import pytest
from scipy.spatial import cKDTree

from fluids_gb300 import capi
from fluids_gb300.scenes import FishTank, jitter, lattice_block

pytestmark = pytest.mark.gpu

DX, BOX = 0.02, (0.8, 0.6, 0.5)
H = 2 * DX


def _context(nbody):
    fluid = jitter(lattice_block(12, 12, 12, DX, (-0.12, -0.12, -0.12)), 0.05 * DX, 1)
    pts = np.ones((nbody, 4), np.float32)
    pts[:, :3] = np.random.default_rng(nbody).uniform(-0.2, 0.2, (nbody, 3))
    ctx = capi.Context(capi.make_params(
        capi.SPH_WCSPH, mode=capi.SPH_MODE_PHYSICS, time_step=1e-6, particle_radius=DX / 2, support_radius=H,
        neigh_cap=100, gas_stiffness=1000.0, surface_tension=0.001, gravity=9.81))
    ctx.set_rect_limits(*BOX)
    ctx.add_boundary(FishTank(*BOX).surface_sampling(DX))
    ctx.add_boundary(pts, can_move=True, mass=2.0)
    ctx.add_volume(fluid)
    return ctx, pts


@pytest.mark.parametrize("nbody", [77_824, 77_825, 155_649])
def test_large_body_force_is_the_pair_sum(gpu_lib, nbody):
    ctx, pts = _context(nbody)
    for s in ("BOUNDARY_SYNC", "HASHES", "SORT", "SHUFFLE", "CELL_INTERVALS", "NEIGH_LIST", "WC_DENSITY"):
        ctx.stage(s)
    pos = ctx.get("POS_SORTED").reshape(-1, 4)[:, :3].astype(np.float64)
    C = ctx.get("PRESSURE").astype(np.float64) / ctx.get("DENSITY").astype(np.float64) ** 2
    phi = ctx.get("BPHI")[-nbody:].astype(np.float64)
    ctx.stage("BOUNDARY_FORCES")
    F, T = ctx.body_forces(2)
    q = pts[:, :3].astype(np.float64)
    near = cKDTree(q).query_ball_tree(cKDTree(pos), H)
    b = np.repeat(np.arange(nbody), [len(k) for k in near])
    f = np.concatenate([np.asarray(k, np.int64) for k in near if k])
    r = pos[f] - q[b]
    n = np.sqrt((r * r).sum(1))
    spiky = -45.0 / (np.pi * np.float64(np.float32(H)) ** 6)
    mass = capi.describe(ctx.params, BOX)["mass"]
    v = r * (mass * phi[b] * 2.0 * C[f] * spiky / n * (H - n) ** 2)[:, None]
    want, tau, size, arm = v.sum(0), np.cross(q[b], v).sum(0), np.abs(v).sum(), np.abs(q).max()
    step, _ = _context(nbody)
    step.simulate(1)
    # float32 terms and sums of at most 100 pairs a particle, then the body's in 256 parts: 1e-5
    # of the terms
    for g, t in ((F, T), step.body_forces(2)):
        assert np.abs(g[1, :3] - want).max() <= 1e-5 * size
        assert np.abs(t[1, :3] - tau).max() <= 2e-5 * size * arm
