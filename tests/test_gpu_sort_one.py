"""The sort's single launch (a tile of pairs per CTA, grid barriers between its phases) and its
limits, against a stable CPU sort: one CTA, a partial last tile, the last size that takes the
launch and the first that does not, one to four digit passes, values that are no identity, and
repeated calls on the same workspace."""
import numpy as np
import pytest
import torch

from fluids_gb300 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 513, 4096, 4097, 6145, 65536, 262145, 524288, 524289])
@pytest.mark.parametrize("bits", [7, 16, 23, 32])
def test_one_launch_sort_is_stable(gpu_lib, n, bits):
    rng = np.random.default_rng(n + bits)
    for top in (1 << bits, 5):   # the whole key range, then nothing but ties
        keys = rng.integers(0, top, size=n, dtype=np.int64).astype(np.uint32)
        vals = rng.integers(-2**31, 2**31, size=n, dtype=np.int64).astype(np.int32)
        dk, dv = torch.from_numpy(keys.view(np.int32)).cuda(), torch.from_numpy(vals).cuda()
        capi.sort_pairs_device(dk.data_ptr(), dv.data_ptr(), n, bits)
        torch.cuda.synchronize()
        order = np.argsort(keys, kind="stable")
        assert np.array_equal(dk.cpu().numpy().view(np.uint32), keys[order])
        assert np.array_equal(dv.cpu().numpy(), vals[order])


def test_sizes_in_turn_share_the_workspace(gpu_lib):
    """A large sort leaves its look-back words in the scratch a small one then uses."""
    rng = np.random.default_rng(3)
    for n in (700_001, 5000, 100, 700_000, 40_001):
        keys = rng.integers(0, 1 << 24, size=n, dtype=np.int64).astype(np.uint32)
        dk = torch.from_numpy(keys.view(np.int32)).cuda()
        dv = torch.arange(n, dtype=torch.int32, device="cuda")
        capi.sort_pairs_device(dk.data_ptr(), dv.data_ptr(), n, 24)
        torch.cuda.synchronize()
        assert np.array_equal(dv.cpu().numpy(), np.argsort(keys, kind="stable").astype(np.int32))
