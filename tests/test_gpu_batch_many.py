"""Batches of many small clouds, on either side of the count up to which the inverse of
the root tiles' ranks is written for every tile of every cloud: grids as the single
calls', and device memory that goes with what the clouds touch."""

import numpy as np
import pytest

from nanovdb_editor import workloads as W

pytestmark = pytest.mark.gpu

NAMES = ("means", "quats", "scales", "opacities", "colors")
VS = 0.01


def _clouds(count, spread):
    """count clouds of one Gaussian inside one leaf (spread 0), or of up to 5 in several root tiles."""
    rng = np.random.default_rng(count)
    clouds = []
    for b in range(count):
        c = W.plain_cloud(1 + (b % 5 if spread else 0), b)
        c["means"] = (np.float32(0.04) + spread * rng.uniform(-60, 60, c["means"].shape)).astype(np.float32)
        c["scales"][:] = np.float32(0.002)
        c["opacities"][:] = np.float32(0.8)
        clouds.append(c)
    return clouds


def _run(ctx, clouds):
    import torch

    allc = W.concat(clouds)
    dev = [torch.from_numpy(np.ascontiguousarray(allc[k])).cuda() for k in NAMES]
    torch.cuda.synchronize()
    start = np.concatenate([[0], np.cumsum([c.n for c in clouds])]).astype(np.int64)
    _, goff, _ = ctx.voxelize_batch(*dev, start, np.full(len(clouds), VS, np.float32))
    return goff


@pytest.mark.parametrize("count", [2, 63, 64, 65, 130])
def test_grids_equal_single_calls(vox_ctx, count):
    clouds = _clouds(count, 1)
    grids = vox_ctx.grids(_run(vox_ctx, clouds))
    for b in {0, 1, count // 2, count - 1}:
        single = vox_ctx.voxelize_host(*[clouds[b][k] for k in NAMES], VS)
        assert np.array_equal(grids[b].buf, single.buf), b


def test_device_memory_of_many_clouds(vox_ctx):
    """1024 clouds of one leaf each.  Besides the grids (a root node is 542 KB), with the buffers'
    margin of an eighth: 9 MB of root bits and prefixes, 9 of lower bits and prefixes (one root
    tile per cloud), 12 of staged values, allocation granules.  32768 words per cloud would be 144."""
    import torch

    from nanovdb_editor.vox import VoxContext

    clouds = _clouds(1024, 0)
    _run(vox_ctx, clouds)  # kernels loaded
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    ctx = VoxContext(0)
    try:
        goff = _run(ctx, clouds)
        torch.cuda.synchronize()
        grew = before - torch.cuda.mem_get_info()[0]
    finally:
        ctx.close()
    assert grew <= 1.125 * int(goff[-1]) + (64 << 20), (grew, int(goff[-1]))
