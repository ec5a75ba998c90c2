"""The reference node order on both sides of the rules that choose its path: one
window of candidates (the canonical order) or several, and a level of up to 2048
nodes (ranked by counting) or more (sorted).  A thin diagonal disc gives the
candidates of a window with few voxels; one Gaussian per lower node the level.
Bit-exact against the oracle's windows."""

import numpy as np
import pytest

from test_gpu_tree import NAMES, VS, _lattice_cloud

pytestmark = pytest.mark.gpu

WINDOW = 8388608


@pytest.mark.parametrize("n", [1900, 2300])
@pytest.mark.parametrize("reach", [45, 95])
def test_order_matches_oracle(vox_ctx, oracle_mod, n, reach):
    from nanovdb_editor.vox import FLAG_WINDOW_ORDER

    c = _lattice_cloud(n, 17, n)
    half = np.pi / 8
    for g in (3, n // 2):
        c["scales"][g] = np.array([reach, reach, 0.3], np.float32) * VS
        c["quats"][g] = np.array([np.cos(half), np.sin(half) / np.sqrt(2), np.sin(half) / np.sqrt(2), 0], np.float32)
        c["opacities"][g] = 0.03
    g = vox_ctx.voxelize_host(*[c[k] for k in NAMES], VS, 0.05, FLAG_WINDOW_ORDER)
    assert (vox_ctx.stats()["candidates"] > WINDOW) == (reach == 95)
    ref = oracle_mod.OracleResult(c, VS, 0.05, window_mode=1)
    assert (ref.counts["lower"] > 2048) == (n == 2300)
    assert np.array_equal(g.node2, ref.node2())
    np.testing.assert_array_equal(g.rgba8, ref.values()["rgba8"])
    ref.close()
