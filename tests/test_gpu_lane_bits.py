"""Sums in list order have the same bits whatever the number of lanes a particle takes: one block of
particles by itself and beside isolated particles far away, as many as each choice of the lanes and
of the list pass begins at (152 SMs).  The isolated ones have no neighbours, so they change neither
the block's lists nor the largest density error of the PCISPH stop test."""
import numpy as np
import pytest

from fluids_gb300 import capi
from fluids_gb300.scenes import FishTank, jitter, lattice_block

pytestmark = pytest.mark.gpu

DX, BOX = 0.012, (4.0, 1.6, 1.6)
SIDE = (13, 17, 11)


def _scene(n):
    """The block in the corner of the tank, then the isolated particles up to n."""
    a = jitter(lattice_block(*SIDE, DX, (-2.0 + DX, -0.8 + DX, -0.8 + DX)), 4e-4, 3)
    g = 2.6 * DX
    far = lattice_block(108, 49, 49, g, (-1.5, -0.75, -0.75))
    p = np.concatenate([a, far[:n - len(a)]]).astype(np.float32)
    assert len(p) == n
    v = np.zeros_like(p)
    v[:len(a), :3] = np.random.default_rng(7).uniform(-0.5, 0.5, (len(a), 3))
    return p, v, len(a)


def _context(p, v, method, walls=True, **kw):
    args = dict(mode=capi.SPH_MODE_PHYSICS, time_step=1e-4, particle_radius=DX / 2, support_radius=2 * DX,
                k_viscosity=0.05, gas_stiffness=2000.0, surface_tension=0.001, gravity=9.81, max_vel=20.0)
    args.update(kw)
    ctx = capi.Context(capi.make_params(method, **args))
    ctx.set_rect_limits(*BOX)
    if walls:
        ctx.add_boundary(FishTank(*BOX).surface_sampling(DX))
    ctx.add_volume(p, v)
    return ctx


def _by_id(ctx, field, count):
    x = ctx.get(field)
    x = x.reshape(len(ctx.get("ID")), -1)
    out = np.empty_like(x)
    out[ctx.get("ID")] = x
    return out[:count]


def _block():
    return SIDE[0] * SIDE[1] * SIDE[2]


def test_pcisph_step(gpu_lib):
    """8 | 4 | 1 lanes (9,728, 38,912); lists by lanes, by pairs of threads (60,800), by one (116,736)."""
    got = []
    for n in (_block(), 9_728, 9_729, 38_912, 38_913, 60_801, 116_737, 200_000):
        p, v, count = _scene(n)
        ctx = _context(p, v, capi.SPH_PCISPH, time_step=5e-4, k_viscosity=1.7, surface_tension=1.0, relax_on_add=0,
                       pcisph_min_iterations=3, pcisph_max_iterations=8, pcisph_error_ratio=0.01)
        for _ in range(2):
            ctx.simulate(1)
        got.append([n, ctx.get("PCI_ITERS")[:1]] + [_by_id(ctx, f, count) for f in (
            "NEIGH_LEN", "SB_NEIGH_LEN", "DENSITY", "NORMAL", "FORCE_OTHER", "PRESSURE", "FORCE_PRESSURE", "POS",
            "VEL")])
        ctx.close()
    assert (got[0][3] > 0).any() and 3 <= got[0][1][0] <= 8
    for other in got[1:]:
        for k, (a, b) in enumerate(zip(got[0][1:], other[1:])):
            assert np.array_equal(a, b), (other[0], k)


@pytest.mark.parametrize("walls", [True, False])
def test_list_and_density_of_a_wcsph_step(gpu_lib, walls):
    """Lanes up to 60,800 (77,824 without walls), pairs of threads up to 116,736, one thread."""
    got = []
    for n in (_block(), 60_800, 60_801, 77_824, 77_825, 116_736, 116_737):
        p, v, count = _scene(n)
        ctx = _context(p, v, capi.SPH_WCSPH, walls)
        ctx.simulate(1)
        got.append([_by_id(ctx, f, count) for f in ("NEIGH_LEN", "SB_NEIGH_LEN", "DENSITY", "PRESSURE")])
        ctx.close()
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert np.array_equal(a, b)


def test_adjoint_forward(gpu_lib):
    """Forces by eight lanes up to 24,320 particles, lists by lanes up to 77,824."""
    got = []
    for n in (_block(), 24_320, 24_321, 77_824, 77_825):
        p, v, count = _scene(n)
        p[:, 0] += 0.5   # away from the container's wall
        ctx = _context(p, v, capi.SPH_WCSPH, False, surface_tension=0.0, gravity=0.0)
        adj = capi.Adjoint(ctx, 4, 2)
        x, u = adj.forward(p, v, 0.05, 2000.0)
        got.append((np.asarray(x).reshape(-1, 4)[:count], np.asarray(u).reshape(-1, 4)[:count]))
        adj.close()
        ctx.close()
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert np.array_equal(a, b)
