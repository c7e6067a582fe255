"""sph_sort_pairs on non-blocking streams: its scratch is the process's, and nothing of a call
may depend on, or run beside, what other streams have queued."""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from fluids_gb300 import capi

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

# the scratch of a sort whose passes need one copy of the pairs, then of one that uses two
MEMORY = """
import torch
from fluids_gb300 import capi
n = 1 << 26
k = torch.randint(0, 1 << 24, (n,), dtype=torch.int32, device="cuda")
v = torch.arange(n, dtype=torch.int32, device="cuda")
capi.sort_pairs_device(k.data_ptr(), v.data_ptr(), 1000, 32)
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
used = []
for bits in (32, 24):
    capi.sort_pairs_device(k.data_ptr(), v.data_ptr(), n, bits)
    torch.cuda.synchronize()
    used.append(free - torch.cuda.mem_get_info()[0])
status = 4 * 256 * 4 * (n // 4096)
slack = 16 << 20
assert used[0] <= 8 * n + status + slack, used
assert used[1] <= 16 * n + status + slack, used
print("held", used)
"""

# captured three-pass sorts on scratch that a four-pass sort laid out
CAPTURED = """
import numpy as np, torch
from fluids_gb300 import capi
rng = np.random.default_rng(2)
n = 700_001
dk = torch.zeros(n, dtype=torch.int32, device="cuda")
dv = torch.zeros(n, dtype=torch.int32, device="cuda")
capi.sort_pairs_device(dk.data_ptr(), dv.data_ptr(), n, 32)
torch.cuda.synchronize()
sizes, graphs = (5_000, 40_001, 300_007, n), []
for m in sizes:
    graphs.append(torch.cuda.CUDAGraph())
    with torch.cuda.graph(graphs[-1]):
        capi.sort_pairs_device(dk.data_ptr(), dv.data_ptr(), m, 24, torch.cuda.current_stream().cuda_stream)
for m, g in list(zip(sizes, graphs)) * 2:
    keys = rng.integers(0, 1 << 24, size=m, dtype=np.int64).astype(np.uint32)
    dk[:m].copy_(torch.from_numpy(keys.view(np.int32)))
    dv[:m].copy_(torch.arange(m, dtype=torch.int32))
    g.replay()
    torch.cuda.synchronize()
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(dv[:m].cpu().numpy(), order.astype(np.int32)), m
    assert np.array_equal(dk[:m].cpu().numpy().view(np.uint32), keys[order]), m
print("replayed")
"""


def _run(code):
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


def test_growing_scratch_beside_a_busy_default_stream(gpu_lib):
    assert "sorted" in _run(BUSY_DEFAULT)


def test_scratch_held(gpu_lib):
    assert "held" in _run(MEMORY)


def test_three_passes_captured_without_a_third_pair(gpu_lib):
    assert "replayed" in _run(CAPTURED)


@pytest.mark.parametrize("n", [65_537, 300_001, 524_288])
def test_barrier_words_left_by_a_timed_out_sort(gpu_lib, n):
    """A cooperative sort whose wait ran out leaves arrivals in its barrier: the next sort on the
    workspace (sph::sort_pairs, as the context's sorts call it) is right all the same."""
    f = getattr(capi.lib(), "_ZN3sph10sort_pairsEP11CUstream_stPjPiS2_S3_iiPvS2_iPS2_PS3_")
    f.restype = None
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 1 << 24, size=n, dtype=np.int64).astype(np.uint32)
    k0 = torch.from_numpy(keys.view(np.int32)).cuda()
    v0 = torch.arange(n, dtype=torch.int32, device="cuda")
    k1, v1 = torch.empty_like(k0), torch.empty_like(v0)
    ws = torch.full((4 * 256 + 64 + 1024 * 256,), 37, dtype=torch.int32, device="cuda")   # barrier words included
    flags = torch.zeros(4, dtype=torch.int32, device="cuda")
    kr, vr = C.c_void_p(), C.c_void_p()
    torch.cuda.synchronize()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    f(C.c_void_p(0), *[C.c_void_p(t.data_ptr()) for t in (k0, v0, k1, v1)], C.c_int(n), C.c_int(24),
      C.c_void_p(ws.data_ptr()), C.c_void_p(flags.data_ptr()), C.c_int(sms), C.byref(kr), C.byref(vr))
    torch.cuda.synchronize()
    assert flags[0].item() == 0
    got = {t.data_ptr(): t for t in (v0, v1)}[vr.value]
    assert np.array_equal(got.cpu().numpy(), np.argsort(keys, kind="stable").astype(np.int32))


@pytest.mark.parametrize("n", [32_769, 200_001, 524_288])
def test_barrier_words_left_before_a_gated_sort(gpu_lib, n):
    """The same for the full sort that the step's sort opens when it has no previous order
    (sph::sort_pairs_incremental), and then its update of that order."""
    lib = capi.lib()
    f = getattr(lib, "_ZN3sph22sort_pairs_incrementalEP11CUstream_stPKjiiPjPiPvS6_S4_iS1_P10CUevent_stS8_b")
    f.restype = None
    size = getattr(lib, "_ZN3sph24sort_inc_workspace_bytesEi")
    size.restype = C.c_size_t
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 1 << 21, size=n, dtype=np.int64).astype(np.uint32)
    inc = torch.zeros(size(C.c_int(n)), dtype=torch.uint8, device="cuda")
    ws = torch.full((4 * 256 + 64 + 1024 * 256,), 37, dtype=torch.int32, device="cuda")
    flags = torch.zeros(4, dtype=torch.int32, device="cuda")
    ko, vo = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for k in range(3):   # no previous order; a few keys moved; most of them moved, so a full sort again
        moved = rng.uniform(size=n) < (0.0, 0.01, 0.9)[k]
        keys = np.where(moved, rng.integers(0, 1 << 21, size=n), keys).astype(np.uint32)
        dk = torch.from_numpy(keys.view(np.int32)).cuda()
        ws[4 * 256 + 32:4 * 256 + 34] = 37
        torch.cuda.synchronize()
        f(C.c_void_p(0), C.c_void_p(dk.data_ptr()), C.c_int(n), C.c_int(21), C.c_void_p(ko.data_ptr()),
          C.c_void_p(vo.data_ptr()), C.c_void_p(inc.data_ptr()), C.c_void_p(ws.data_ptr()), C.c_void_p(flags.data_ptr()),
          C.c_int(sms), C.c_void_p(0), C.c_void_p(0), C.c_void_p(0), C.c_bool(False))
        torch.cuda.synchronize()
        order = np.argsort(keys, kind="stable")
        assert flags[0].item() == 0
        assert np.array_equal(vo.cpu().numpy(), order.astype(np.int32)), k
        keys = keys[order]   # the step hands the next call its particles in this order


@pytest.mark.parametrize("sizes", [(3_000, 4_000), (30_000, 20_001), (65_536, 40_000), (300_007, 150_001),
                                   (700_001, 5_000)])
def test_two_streams_share_the_scratch(gpu_lib, sizes):
    """Sorts on two non-blocking streams, queued without waiting: each waits on the GPU for the one
    before it, although a small sort's launch may be set up early."""
    rng = np.random.default_rng(sizes[0])
    streams = [torch.cuda.Stream() for _ in sizes]
    keys = [rng.integers(0, 1 << 24, size=n, dtype=np.int64).astype(np.uint32) for n in sizes]
    first = [torch.from_numpy(k.view(np.int32)).cuda() for k in keys]
    rounds = [[(a.clone(), torch.arange(len(a), dtype=torch.int32, device="cuda")) for a in first] for _ in range(12)]
    big = max(range(2), key=lambda i: sizes[i])
    k0, v0 = first[big].clone(), torch.arange(sizes[big], dtype=torch.int32, device="cuda")
    capi.sort_pairs_device(k0.data_ptr(), v0.data_ptr(), sizes[big], 24)   # the scratch
    torch.cuda.synchronize()
    for pairs in rounds:
        for (dk, dv), s in zip(pairs, streams):
            capi.sort_pairs_device(dk.data_ptr(), dv.data_ptr(), len(dk), 24, s.cuda_stream)
    torch.cuda.synchronize()
    for pairs in rounds:
        for (dk, dv), k in zip(pairs, keys):
            order = np.argsort(k, kind="stable")
            assert np.array_equal(dv.cpu().numpy(), order.astype(np.int32))
            assert np.array_equal(dk.cpu().numpy().view(np.uint32), k[order])
