"""The sort by several launches where its warps choose between two ways to match digits: keys of few
digits a warp, of many, and of warps whose first round (by which they choose) is unlike the others,
at the first size of that path and with a partial last tile."""
import numpy as np
import pytest
import torch

from fluids_gb300 import capi

pytestmark = pytest.mark.gpu


def _keys(kind, n, bits, rng):
    k = rng.integers(0, 1 << bits, size=n, dtype=np.int64)
    first = (np.arange(n) // 32) % 16 == 0   # the first of a warp's sixteen rounds
    if kind == "sorted":
        k = np.sort(k)
    elif kind == "near":
        k = np.where(rng.uniform(size=n) < 0.02, k, np.sort(k))
    elif kind == "nine":
        k = (k % 9) * ((1 << bits) // 9)
    elif kind == "equal first":
        k = np.where(first, (1 << bits) - 1, k)
    elif kind == "equal after":
        k = np.where(first, k, 3)
    return k.astype(np.uint32)


@pytest.mark.parametrize("kind", ["sorted", "near", "nine", "equal first", "equal after"])
@pytest.mark.parametrize("n,bits", [(524_289, 8), (700_001, 16), (700_001, 24), (1_500_007, 32)])
def test_digits_few_and_many(gpu_lib, kind, n, bits):
    keys = _keys(kind, n, bits, np.random.default_rng(bits))
    order = np.argsort(keys, kind="stable").astype(np.int32)
    dk = torch.from_numpy(keys.view(np.int32)).cuda()
    dv = torch.arange(n, dtype=torch.int32, device="cuda")
    capi.sort_pairs_device(dk.data_ptr(), dv.data_ptr(), n, bits)
    torch.cuda.synchronize()
    assert np.array_equal(dv.cpu().numpy(), order)
    assert np.array_equal(dk.cpu().numpy().view(np.uint32), keys[order])
