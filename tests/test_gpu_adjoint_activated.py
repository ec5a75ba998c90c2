"""The adjoint with respect to activated inputs, whose quaternions are used as given:
the rotation is orthogonal for unit quaternions only, and singular where w = 0 and
|v|^2 = 1/2.  Against the oracle's FP64 adjoint, within 1e-5 of each family's maximum."""

import numpy as np
import pytest

from nanovdb_editor import workloads as W
from test_gpu_adjoint import NAMES, REL
from test_oracle_adjoint import upstream

pytestmark = pytest.mark.gpu


def _activated(kind, n, vs):
    rng = np.random.default_rng(n)
    c = W.plain_cloud(n, n + 3)
    c["means"] = rng.uniform(-12 * vs, 12 * vs, (n, 3)).astype(np.float32)
    c["scales"] = (vs * np.exp(rng.uniform(np.log(0.2), np.log(3.0), (n, 3)))).astype(np.float32)
    c["opacities"] = rng.uniform(0.2, 0.95, n).astype(np.float32)
    q = rng.standard_normal((n, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    if kind == "norm":
        q *= rng.uniform(0.5, 2.0, (n, 1))
    elif kind == "singular":
        q[:, 0] = 0.0
        q *= np.sqrt(0.5) / np.linalg.norm(q, axis=1, keepdims=True)
        q[n // 2 :] += rng.uniform(-1e-3, 1e-3, (n - n // 2, 4))
    c["quats"] = q.astype(np.float32)
    return {k: np.ascontiguousarray(c[k]) for k in NAMES}


@pytest.mark.parametrize("n", [1, 33, 900])
@pytest.mark.parametrize("kind", ["unit", "bf16", "norm", "singular"])
def test_backward_of_activated_inputs(vox_ctx, oracle_mod, kind, n):
    import torch

    from nanovdb_editor.vox import FLAG_BF16_INPUTS, FLAG_DIFFERENTIABLE

    vs = 0.01
    params = _activated(kind, n, vs)
    dev = {k: torch.from_numpy(v).cuda() for k, v in params.items()}
    flags = FLAG_DIFFERENTIABLE
    if kind == "bf16":  # every attribute, stored so
        dev = {k: v.to(torch.bfloat16) for k, v in dev.items()}
        params = {k: v.float().cpu().numpy() for k, v in dev.items()}
        flags |= FLAG_BF16_INPUTS
    torch.cuda.synchronize()
    ref = oracle_mod.OracleResult(params, vs, 0.05, window_mode=oracle_mod.OV_MODE_SMOOTH)
    vox_ctx.voxelize(*[dev[k] for k in NAMES], vs, 0.05, flags)
    vc = ref.counts["value_count"]
    assert int(vox_ctx.stats()["value_count"]) == vc
    gd, gc = (a.astype(np.float32) for a in upstream(vc, n))
    out = {k: torch.empty(dev[k].shape, dtype=torch.float32, device="cuda") for k in NAMES}
    vox_ctx.backward(*[dev[k] for k in NAMES], torch.from_numpy(gd).cuda(), torch.from_numpy(gc).cuda(), out)
    an = ref.smooth_grad64(params, False, gd.astype(np.float64), gc.astype(np.float64))
    for k in NAMES:
        scale = float(np.abs(an[k]).max())
        err = float(np.abs(out[k].cpu().numpy().astype(np.float64).reshape(an[k].shape) - an[k]).max())
        assert scale > 0 and err <= REL * scale, (k, err / scale)
    ref.close()
