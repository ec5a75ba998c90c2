"""The 64-bit scan at the edges of its tiles (2048 elements) and of its warp-wide
look-back (32 tiles per step), with 16-byte aligned arrays and arrays 8 bytes
off, in place and out of place, with sums that wrap mod 2^64."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 2047, 2048, 2049, 2 * 2048, 32 * 2048, 33 * 2048 - 1, 33 * 2048 + 1, 700 * 2048 + 3])
@pytest.mark.parametrize("skip", [0, 1])
@pytest.mark.parametrize("inclusive", [True, False])
def test_scan_matches_numpy(vox_ctx, n, skip, inclusive):
    import torch

    rng = np.random.default_rng(n * 4 + skip * 2 + inclusive)
    x = rng.integers(0, 1 << 63, n, dtype=np.uint64) * np.uint64(2) + np.uint64(1)
    want = np.cumsum(x, dtype=np.uint64)
    total = int(want[-1])
    if not inclusive:
        want = want - x
    buf = torch.zeros(n + 2, dtype=torch.int64, device="cuda")
    out = torch.full((n + 2,), -7, dtype=torch.int64, device="cuda")
    tot = torch.zeros(1, dtype=torch.int64, device="cuda")
    buf[skip:skip + n] = torch.from_numpy(x.view(np.int64)).cuda()
    for dst in (out, buf):
        torch.cuda.synchronize()
        vox_ctx.global_scan_u64(buf[skip:skip + n], dst[skip:skip + n], tot, inclusive)
        np.testing.assert_array_equal(dst[skip:skip + n].cpu().numpy().view(np.uint64), want)
        assert int(tot.cpu().numpy().view(np.uint64)[0]) == total
    assert (out[:skip] == -7).all() and (out[skip + n:] == -7).all()
