"""A batch that is large enough for the tiled passes (above 116,736 particles on 152 SMs), with
partial last tiles: every shape of the grid, among them ones whose few warps stride over many tiles,
gives the same state bit for bit, and each scene's is that of its own context."""
import numpy as np
import pytest

from fluids_gb300 import capi, workloads

pytestmark = pytest.mark.gpu

SHAPES = ((256, 0), (32, 1), (64, 1), (256, 1), (128, 3))


@pytest.mark.parametrize("sigma", [0.001, 0.0])
def test_tile_shapes_of_a_large_batch(gpu_lib, sigma):
    scenes = workloads.batched_scenes(14, seed=4, nmin=3000, nmax=30000)
    total = sum(len(s["fluid"]) for s in scenes)
    assert total > 116_736 and sum(len(s["fluid"]) % 32 != 0 for s in scenes) >= 5
    shared = workloads.wcsph_params(0.015, 2e-4, sigma=sigma)
    out, strides = [], 0
    for bs, ctas in SHAPES:
        batch = capi.BatchContext(shared, scenes)
        batch.set_block_size(bs)
        batch.set_tile_shape(ctas)
        sh = batch.tile_shape()
        strides += sh["tiles"] > 3 * sh["blocks"] * (bs // 32)
        batch.simulate(3)
        out.append([batch.get(f) for f in ("POS", "VEL", "NEIGH_LEN", "DENSITY", "ID")])
        assert batch.device_flags() & (capi.FLAGS["NAN"] | capi.FLAGS["TIMEOUT"]) == 0
        ranges = [batch.scene_range(k) for k in range(len(scenes))]
        batch.close()
    assert strides >= 3   # shapes whose warps take more than three tiles each
    for o in out[1:]:
        for a, b in zip(out[0], o):
            assert np.array_equal(a, b)
    pos = out[0][0].reshape(-1, 4)[:, :3]
    for k in (0, 5, 13):
        single = workloads.build_scene_context(shared, scenes[k])
        single.simulate(3)
        first, count = ranges[k]
        a = np.empty((count, 3)), np.empty((count, 3))
        a[0][out[0][4][first:first + count] - first] = pos[first:first + count]
        a[1][single.get("ID")] = single.get("POS").reshape(-1, 4)[:, :3]
        # three steps of float32 sums in another order, as the other tests of a batch
        assert np.abs(a[0] - a[1]).max() <= 1e-5
        single.close()
