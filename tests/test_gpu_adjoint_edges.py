"""The adjoint where its warps and batches end: pair counts around 32, boxes of one
column, of more columns than lanes and of whole leaves (a batch then holds two), and
pairs of several leaves in one batch.  Against the oracle's FP64 adjoint, within 1e-5
of each family's maximum."""

import numpy as np
import pytest

from nanovdb_editor import workloads as W
from test_gpu_adjoint import NAMES, REL, _dev, _gpu_grads
from test_oracle_adjoint import raw_params, smooth_forward, upstream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 130])
@pytest.mark.parametrize("kind", ["point", "wide", "mixed"])
def test_backward_edges(vox_ctx, oracle_mod, kind, n):
    vs = 0.01
    rng = np.random.default_rng(n)
    c = W.plain_cloud(n, n + 7)
    lo, hi = {"point": (0.05, 0.4), "wide": (3.0, 6.0), "mixed": (0.1, 5.0)}[kind]
    c["means"] = rng.uniform(-6 * vs, 6 * vs, (n, 3)).astype(np.float32)
    c["scales"] = (vs * np.exp(rng.uniform(np.log(lo), np.log(hi), (n, 3)))).astype(np.float32)
    c["opacities"] = rng.uniform(0.3, 0.95, n).astype(np.float32)
    params = raw_params(c, n)
    ref = smooth_forward(oracle_mod, params, vs)
    gd64, gc64 = upstream(ref.counts["value_count"], n)
    gd, gc = gd64.astype(np.float32), gc64.astype(np.float32)
    got = _gpu_grads(vox_ctx, _dev(params), vs, gd, gc)
    an = ref.smooth_grad64(params, True, gd.astype(np.float64), gc.astype(np.float64))
    for k in NAMES:
        scale = float(np.abs(an[k]).max())
        err = float(np.abs(got[k].reshape(an[k].shape) - an[k]).max())
        assert err <= REL * max(scale, 1e-30), (k, err, scale)
    ref.close()
