"""The forces on a body's particles with several lanes a particle, against the pair sum in
float64 from the fields they read: bodies of one particle, a partial warp and block, dense
cells, and the per-particle cap; and the step's body streams against the stage path."""
import numpy as np
import pytest

from fluids_gb300 import capi
from fluids_gb300.scenes import FishTank, jitter, lattice_block

pytestmark = pytest.mark.gpu

DX, BOX = 0.02, (0.8, 0.6, 0.5)


def _context(nbody, crowd, cap=50, seed=0, **kw):
    rng = np.random.default_rng(seed + nbody)
    d = DX / crowd ** (1.0 / 3.0)
    k = int(0.3 / d)
    fluid = jitter(lattice_block(k, k, k, d, (-0.15, -0.15, -0.15)), 0.1 * d, seed)
    pts = np.ones((nbody, 4), np.float32)
    pts[:, :3] = rng.uniform(-0.12, 0.12, (nbody, 3))
    p = capi.make_params(capi.SPH_WCSPH, mode=capi.SPH_MODE_PHYSICS, time_step=1e-5, particle_radius=DX / 2,
                         support_radius=2 * DX, neigh_cap=cap, gas_stiffness=1000.0, surface_tension=0.001,
                         gravity=9.81, **kw)
    ctx = capi.Context(p)
    ctx.set_rect_limits(*BOX)
    ctx.add_boundary(FishTank(*BOX).surface_sampling(DX))
    ctx.add_boundary(pts, can_move=True, mass=2.0)
    ctx.set_body_dynamics(1, True, (1.0, 1.0, 1.0), 0.0)
    ctx.add_volume(fluid)
    return ctx, pts


@pytest.mark.parametrize("nbody,crowd", [(1, 1), (5, 1), (33, 1), (300, 1), (40, 1.4)])
def test_body_force_is_the_pair_sum(gpu_lib, nbody, crowd):
    ctx, pts = _context(nbody, crowd, cap=100)
    for s in ("BOUNDARY_SYNC", "HASHES", "SORT", "SHUFFLE", "CELL_INTERVALS", "NEIGH_LIST", "WC_DENSITY"):
        ctx.stage(s)
    pos = ctx.get("POS_SORTED").reshape(-1, 4)[:, :3].astype(np.float64)
    C = ctx.get("PRESSURE").astype(np.float64) / ctx.get("DENSITY").astype(np.float64) ** 2
    phi = ctx.get("BPHI")[-nbody:].astype(np.float64)
    d = capi.describe(ctx.params, BOX)
    H = 2 * DX
    ctx.stage("BOUNDARY_FORCES")
    F, T = ctx.body_forces(2)
    spiky = -45.0 / (np.pi * np.float64(np.float32(H)) ** 6)
    want, tau, size, arm = np.zeros(3), np.zeros(3), 0.0, 0.0
    for q, f in zip(pts[:, :3].astype(np.float64), phi):
        r = pos - q
        n = np.sqrt((r * r).sum(1))
        w = n < H
        v = (d["mass"] * f) * (r[w] * (2.0 * C[w] * spiky / n[w] * (H - n[w]) ** 2)[:, None])
        want += v.sum(0)
        tau += np.cross(q, v.sum(0))
        size += np.abs(v).sum()
        arm = max(arm, np.linalg.norm(q))
    # float32 terms and sums of at most 100 pairs a particle, then the body's: 1e-5 of the terms
    assert np.abs(F[1, :3] - want).max() <= 1e-5 * size
    assert np.abs(T[1, :3] - tau).max() <= 1e-5 * size * arm
    assert not F[0].any()


def test_body_streams_equal_the_stages(gpu_lib):
    """Three steps with the body's passes beside the fluid's, with and without a graph, against
    the stages one after the other."""
    stages = ("BOUNDARY_SYNC", "HASHES", "SORT", "SHUFFLE", "CELL_INTERVALS", "NEIGH_LIST", "WC_DENSITY",
              "BOUNDARY_FORCES", "NORMALS", "WC_ACCEL", "WC_INTEGRATE")
    ctxs = [_context(200, 1, use_graph=g)[0] for g in (1, 0, 0)]
    for c in ctxs[:2]:
        c.simulate(3)
    for _ in range(3):
        for s in stages:
            ctxs[2].stage(s)
    want = ctxs[2].body_state(1)
    for c in ctxs[:2]:
        for x, y in zip(c.body_state(1), want):
            assert np.abs(x - y).max() <= 1e-5 * max(1.0, np.abs(y).max())
        x, y = (k.get("POS").reshape(-1, 4)[:, :3] for k in (c, ctxs[2]))
        assert np.abs(x - y).max() <= 1e-6
    assert np.array_equal(ctxs[0].get("POS"), ctxs[1].get("POS"))
