"""sph_sort_pairs on non-blocking streams: its scratch is the process's, and nothing of a call
may depend on, or run beside, what other streams have queued."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# a first and two growing calls: one cluster, one cooperative launch, several launches
BUSY_DEFAULT = """
import numpy as np, torch
from fluids_gb300 import capi
rng = np.random.default_rng(5)
side = torch.cuda.Stream()
for n in (50_001, 300_007, 700_001):
    keys = rng.integers(0, 1 << 24, size=n, dtype=np.int64).astype(np.uint32)
    dk = torch.from_numpy(keys.view(np.int32)).cuda()
    dv = torch.arange(n, dtype=torch.int32, device="cuda")
    order = np.argsort(keys, kind="stable")
    torch.cuda.synchronize()
    for cycles in (2_000_000, 200_000_000):   # about 1 ms, then about 100 ms
        torch.cuda._sleep(cycles)
        capi.sort_pairs_device(dk.data_ptr(), dv.data_ptr(), n, 24, side.cuda_stream)
        side.synchronize()
        assert np.array_equal(dk.cpu().numpy().view(np.uint32), keys[order]), n
        assert np.array_equal(dv.cpu().numpy(), order.astype(np.int32)), n
        torch.cuda.synchronize()
        dk.copy_(torch.from_numpy(keys.view(np.int32)))
        dv.copy_(torch.arange(n, dtype=torch.int32))
        torch.cuda.synchronize()
print("sorted")
"""


def _run(code):
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


def test_growing_scratch_beside_a_busy_default_stream(gpu_lib):
    assert "sorted" in _run(BUSY_DEFAULT)
