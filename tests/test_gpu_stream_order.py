"""Voxel coordinates are written on the library's own stream into a tensor that
torch fills first: with torch's stream held up by earlier work the fill must
still come first."""

import numpy as np
import pytest

from nanovdb_editor import workloads as W

pytestmark = pytest.mark.gpu

NAMES = ("means", "quats", "scales", "opacities", "colors")


def _busy(torch):
    a = torch.ones(4096, 4096, device="cuda")
    for _ in range(40):
        a = a @ a * 1e-4
    return a


@pytest.mark.parametrize("batch", [False, True])
def test_coords_follow_the_fill(vox_ctx, batch):
    import torch

    from nanovdb_editor.autograd import batch_voxel_keys, voxel_coords

    vs = 0.01
    c = W.plain_cloud(3000, 5)
    dev = [torch.from_numpy(c[k]).cuda() for k in NAMES]
    torch.cuda.synchronize()
    if batch:
        _, _, voff = vox_ctx.voxelize_batch(*dev, np.array([0, 1200, 3000], np.int64), np.array([vs, vs], np.float32), 0.05, 0)
        want_keys, want_valid = batch_voxel_keys(vox_ctx, voff, "cuda")
        torch.cuda.synchronize()
        hold = _busy(torch)
        keys, valid = batch_voxel_keys(vox_ctx, voff, "cuda")
        assert torch.equal(keys, want_keys) and torch.equal(valid, want_valid)
        assert torch.unique(keys[valid]).numel() == int(valid.sum()) > 1000
    else:
        vox_ctx.voxelize(*dev, vs)
        count = vox_ctx.grid().value_count
        want = torch.empty(count, 3, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        vox_ctx.voxel_coords(want)
        hold = _busy(torch)
        assert torch.equal(voxel_coords(vox_ctx, count, "cuda"), want[2:])
    del hold
