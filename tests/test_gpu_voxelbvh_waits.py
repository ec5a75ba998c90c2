"""The VoxelBVH range pass when its bounded look-back gives up: with every publication
withheld, a run of equal keys that goes on past its tile leaves the last tile without a
run start and with an empty prefix.  The call returns VOX_ERR_TIMEOUT, and no word
beside the caller's arrays changes.  The sort is fixed to the shape without look-back
and the slots' scan has one tile, so this wait is the only one that expires."""

from ctypes import byref, c_int64

import numpy as np
import pytest

from nanovdb_editor import workloads as W

pytestmark = pytest.mark.gpu

GUARD = 64  # words on either side of each array
FILL = 0x5A5A5A5A


# all Gaussians but one at the box's upper corner, in 4 or 8 cells each (unused slots, or none)
@pytest.mark.parametrize("scale", [0.01, 0.02])
@pytest.mark.parametrize("n", [1300, 2047])
def test_ranges_wait_expires_within_bounds(vox_ctx, oracle_mod, monkeypatch, n, scale):
    import torch

    from nanovdb_editor.vox import STATUS, VoxContext, _ptr

    cloud = W.plain_cloud(n, 9)
    cloud["means"][:] = np.float32(0.5)
    cloud["means"][0] = -0.5
    cloud["quats"][:] = np.array([1, 0, 0, 0], np.float32)
    cloud["scales"][:] = np.float32(scale)
    cloud["opacities"][:] = np.float32(0.9)
    ref = oracle_mod.voxelbvh_ijkl(cloud, 64)
    used = int((ref["ijkl"] != np.uint64(0xFFFFFFFFFFFFFFFF)).sum())
    starts = ref["range"].reshape(-1, 2)[: ref["ranges"], 0]
    last_tile = (used - 1) // 2048 * 2048
    assert last_tile > 0 and not (starts[starts < used] >= last_tile).any()  # no run starts in the last tile
    monkeypatch.setenv("VOX_SORT_SHAPE", "5")
    ctx = VoxContext(0)
    try:
        ins = [torch.from_numpy(np.ascontiguousarray(cloud[k], dtype=np.float32)).cuda()
               for k in ("means", "opacities", "quats", "scales")]
        words = {"ijkl": 16 * n, "prim_id": 8 * n, "range": 16 * n}

        def run():
            bufs = {k: torch.full((w + 2 * GUARD,), FILL, dtype=torch.int32, device="cuda") for k, w in words.items()}
            box = torch.empty(6, dtype=torch.float32, device="cuda")
            count = c_int64(-1)
            torch.cuda.synchronize()
            rc = ctx.lib.vox_voxelbvh_ijkl_from_gaussians(ctx.handle, *[_ptr(a) for a in ins], n, 64, 0,
                                                          *[_ptr(bufs[k][GUARD:]) for k in words], _ptr(box), byref(count))
            torch.cuda.synchronize()
            for k, b in bufs.items():
                assert bool((b[:GUARD] == FILL).all()) and bool((b[-GUARD:] == FILL).all()), k
            return rc, {k: b[GUARD:-GUARD].cpu().numpy().copy() for k, b in bufs.items()}, count.value

        ctx.set_wait_limit(1000, withhold_publication=True)
        rc, _, _ = run()
        assert STATUS[rc] == "bounded device wait expired"
        ctx.set_wait_limit(None)
        rc, got, count = run()
        assert rc == 0 and count == ref["ranges"]
        np.testing.assert_array_equal(got["ijkl"].view(np.uint64), ref["ijkl"])
        np.testing.assert_array_equal(got["prim_id"].view(np.uint32), ref["prim_id"])
        np.testing.assert_array_equal(got["range"].view(np.uint32), ref["range"])
    finally:
        ctx.close()
