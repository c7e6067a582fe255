"""The per-particle cap of the forces on bodies: the pair sum in float64 over the first cap
neighbours in cell and list order, by several lanes a particle and (above 77,824 particles of bodies
with mass on 152 SMs) by one thread."""
import numpy as np
import pytest

from fluids_gb300 import capi
from fluids_gb300.scenes import FishTank, jitter, lattice_block

pytestmark = pytest.mark.gpu

DX, BOX = 0.02, (0.8, 0.6, 0.5)
H = np.float32(2 * DX)
OFFSETS = [(0, 0, 0)] + [(x, y, z) for x in (-1, 0, 1) for y in (-1, 0, 1) for z in (-1, 0, 1) if (x, y, z) != (0, 0, 0)]


@pytest.mark.parametrize("cap", [1, 5, 17])
@pytest.mark.parametrize("far", [0, 77_800])
def test_forces_take_the_first_cap_pairs(gpu_lib, cap, far):
    fluid = jitter(lattice_block(12, 12, 12, DX, (-0.12, -0.12, -0.12)), 0.1 * DX, 2)
    rng = np.random.default_rng(cap)
    near = np.ones((60, 4), np.float32)
    near[:, :3] = rng.uniform(-0.1, 0.1, (60, 3))
    pts = np.concatenate([near, np.ones((far, 4), np.float32)])
    pts[60:, :3] = rng.uniform(-0.02, 0.02, (far, 3)) + (0.3, 0.2, 0.2)   # no fluid there
    ctx = capi.Context(capi.make_params(
        capi.SPH_WCSPH, mode=capi.SPH_MODE_PHYSICS, time_step=1e-5, particle_radius=DX / 2, support_radius=2 * DX,
        neigh_cap=cap, gas_stiffness=1000.0, surface_tension=0.001, gravity=9.81))
    ctx.set_rect_limits(*BOX)
    ctx.add_boundary(FishTank(*BOX).surface_sampling(DX))
    ctx.add_boundary(pts, can_move=True, mass=2.0)
    ctx.add_volume(fluid)
    for s in ("BOUNDARY_SYNC", "HASHES", "SORT", "SHUFFLE", "CELL_INTERVALS", "NEIGH_LIST", "WC_DENSITY"):
        ctx.stage(s)
    pos = ctx.get("POS_SORTED").reshape(-1, 4)[:, :3]
    rho = np.float32(1000.0) + np.arange(len(pos), dtype=np.float32) % 7   # densities and pressures of their own
    p = 1e3 + 10.0 * (np.arange(len(pos), dtype=np.float32) % 11)
    ctx.set("DENSITY", rho)
    ctx.set("PRESSURE", p.astype(np.float32))
    phi = ctx.get("BPHI")[-len(pts):].astype(np.float64)
    tab = ctx.get("CELL_INTERVALS").reshape(-1, 2)
    d = capi.describe(ctx.params, BOX)
    origin, dims = np.asarray(d["grid_origin"], np.float32), d["grid_dims"]
    ctx.stage("BOUNDARY_FORCES")
    F, _ = ctx.body_forces(2)
    C = p.astype(np.float64) / rho.astype(np.float64) ** 2
    spiky = -45.0 / (np.pi * np.float64(H) ** 6)
    want, size, most = np.zeros(3), 0.0, 0
    for q, f in zip(near[:, :3], phi):
        cell = np.floor((q - origin) / H).astype(int)
        kept = []
        for o in OFFSETS:
            x, y, z = cell + o
            a, b = tab[x + dims[0] * (y + dims[1] * z)]
            for j in range(a, b):
                r = pos[j] - q
                if (r * r).sum() < H * H:
                    kept.append(j)
        most = max(most, len(kept))
        kept = kept[:cap]
        r = pos[kept].astype(np.float64) - q.astype(np.float64)
        n = np.sqrt((r * r).sum(1))
        v = (d["mass"] * f) * (r * (2.0 * C[kept] * spiky / n * (H - n) ** 2)[:, None])
        want += v.sum(0)
        size += np.abs(v).sum()
    assert most > 17   # the cap cuts
    # float32 terms and sums of at most 17 pairs a particle, then the body's: 1e-5 of the terms
    assert np.abs(F[1, :3] - want).max() <= 1e-5 * size
