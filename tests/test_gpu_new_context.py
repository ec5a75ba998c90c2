"""A new context's first waits: its page-locked words may be a closed context's, whose
publication numbers started at 1 too.  The closed context published exactly once (a
call that failed at its first wait, or one scan), so a new context that took its word
for its own would go on with that context's counts before its kernels had run."""

import numpy as np
import pytest

from nanovdb_editor import workloads as W

pytestmark = pytest.mark.gpu

NAMES = ("means", "quats", "scales", "opacities", "colors")


def _failed_call(ctx):
    from nanovdb_editor.exceptions import PipelineError

    far = W.plain_cloud(300, 5)
    far["means"][7] = 1e6
    with pytest.raises(PipelineError):
        ctx.voxelize_host(*[far[k] for k in NAMES], 0.01)


def _one_scan(ctx):
    import torch

    x = torch.arange(5000, dtype=torch.int64, device="cuda")
    out, total = torch.empty_like(x), torch.zeros(1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    ctx.global_scan_u64(x, out, total, True)
    assert int(total) == 4999 * 5000 // 2


@pytest.mark.parametrize("first", [_failed_call, _one_scan])
def test_context_after_one_publication(vox_ctx, first):
    from nanovdb_editor.vox import VoxContext

    clouds = [W.plain_cloud(n, 60 + i) for i, n in enumerate((1, 4000, 40))]
    want = [vox_ctx.voxelize_host(*[c[k] for k in NAMES], 0.01).buf.copy() for c in clouds]
    for _ in range(4):
        for c, w in zip(clouds, want):
            old = VoxContext(0)
            first(old)
            old.close()
            new = VoxContext(0)
            try:
                assert np.array_equal(new.voxelize_host(*[c[k] for k in NAMES], 0.01).buf, w)
            finally:
                new.close()
