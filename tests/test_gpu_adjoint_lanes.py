"""One forward step of the differentiable solver against the stage path's one-thread passes, at
sizes on both sides of the rules of its list pass (77,824 particles on 152 SMs) and of its force
pass (24,320)."""
import numpy as np
import pytest

from fluids_gb300 import capi, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 24320, 24321, 77824, 77825])
def test_forward_step_equals_one_thread_passes(gpu_lib, n):
    w = workloads.adjoint_block(int(np.ceil(n ** (1.0 / 3.0))), steps=4)
    rng = np.random.default_rng(n)
    w["fluid"] = np.ascontiguousarray(w["fluid"][:n])
    w["velocities"] = np.zeros_like(w["fluid"])
    w["velocities"][:, :3] = rng.uniform(-0.5, 0.5, (n, 3))
    a, b = workloads.build_context(w), workloads.build_context(w)
    adj = capi.Adjoint(a, 1, 1)
    xT, vT = adj.forward(w["fluid"], w["velocities"], w["mu"], w["kgas"])
    assert adj.flags() == 0
    for s in ("HASHES", "SORT", "SHUFFLE", "CELL_INTERVALS", "NEIGH_LIST", "WC_DENSITY", "WC_ACCEL", "WC_INTEGRATE"):
        b.stage(s)
    ids = b.get("ID")
    # the same sums of at most 50 terms, with reciprocals of the density in place of divisions: the
    # parity bar of the float fields, 1e-5 of the largest value
    for f, got, rtol in (("POS", xT, 1e-6), ("VEL", vT, 1e-5)):
        y = np.empty((n, 3))
        y[ids] = b.get(f).reshape(-1, 4)[:, :3]
        assert np.abs(got[:, :3].astype(np.float64) - y).max() <= rtol * np.abs(y).max()
