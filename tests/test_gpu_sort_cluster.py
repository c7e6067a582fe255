"""The sort as one cluster (up to 16 tiles of 2,048 pairs, then of 4,096) at the edges of its
rules, against a stable CPU sort, eagerly and replayed from a captured graph."""
import numpy as np
import pytest
import torch

from fluids_gb300 import capi

pytestmark = pytest.mark.gpu


def _check(dk, dv, keys):
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(dk.cpu().numpy().view(np.uint32), keys[order])
    assert np.array_equal(dv.cpu().numpy(), order.astype(np.int32))


@pytest.mark.parametrize("n", [2, 4097, 6144, 14337, 16384, 16385, 32767, 32768, 32769, 36865, 65535, 65536, 65537])
@pytest.mark.parametrize("bits", [8, 21, 32])
def test_cluster_sort_is_stable(gpu_lib, n, bits):
    rng = np.random.default_rng(n + bits)
    for top in (1 << bits, 3):
        keys = rng.integers(0, top, size=n, dtype=np.int64).astype(np.uint32)
        dk = torch.from_numpy(keys.view(np.int32)).cuda()
        dv = torch.arange(n, dtype=torch.int32, device="cuda")
        capi.sort_pairs_device(dk.data_ptr(), dv.data_ptr(), n, bits)
        torch.cuda.synchronize()
        _check(dk, dv, keys)


@pytest.mark.parametrize("n", [1000, 20000, 50000])
def test_cluster_sort_in_a_captured_graph(gpu_lib, n):
    rng = np.random.default_rng(n)
    dk = torch.zeros(n, dtype=torch.int32, device="cuda")
    dv = torch.zeros(n, dtype=torch.int32, device="cuda")
    capi.sort_pairs_device(dk.data_ptr(), dv.data_ptr(), n, 24)   # the scratch, outside the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        capi.sort_pairs_device(dk.data_ptr(), dv.data_ptr(), n, 24, torch.cuda.current_stream().cuda_stream)
    for _ in range(2):
        keys = rng.integers(0, 1 << 24, size=n, dtype=np.int64).astype(np.uint32)
        dk.copy_(torch.from_numpy(keys.view(np.int32)))
        dv.copy_(torch.arange(n, dtype=torch.int32))
        graph.replay()
        torch.cuda.synchronize()
        _check(dk, dv, keys)
