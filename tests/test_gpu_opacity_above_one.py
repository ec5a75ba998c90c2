"""Activated opacities above 1, which the library takes as given: near such a
Gaussian's centre the base 1 - a of the opacity transform is negative, and the float channels'
alpha is 0 there.  Those channels against the oracle, bit for bit, at exponents from
far below 1 (large Gaussians) to far above."""

import numpy as np
import pytest

from nanovdb_editor import workloads as W

pytestmark = pytest.mark.gpu

NAMES = ("means", "quats", "scales", "opacities", "colors")


@pytest.mark.parametrize("opacity", [1.0, 1.0000001, 1.05, 1.5, 40.0])
@pytest.mark.parametrize("size", [0.3, 1.5, 8.0])  # scale / voxel
@pytest.mark.parametrize("every", [1, 3])  # alone, or among opacities below 1
def test_float_channels(vox_ctx, oracle_mod, opacity, size, every):
    vs, n = 0.01, 150
    rng = np.random.default_rng(n)
    c = W.plain_cloud(n, 81)
    c["means"] = rng.uniform(-10 * vs, 10 * vs, (n, 3)).astype(np.float32)
    c["scales"] = (vs * size * rng.uniform(0.5, 1.5, (n, 3))).astype(np.float32)
    c["opacities"] = rng.uniform(0.2, 0.95, n).astype(np.float32)
    c["opacities"][::every] = np.float32(opacity)
    g = vox_ctx.voxelize_host(*[c[k] for k in NAMES], vs, 1.0)
    ref = oracle_mod.OracleResult(c, vs, 1.0, window_mode=0)
    assert ref.counts["error"] == 0 and ref.counts["V"] > 0
    v = ref.values()
    np.testing.assert_array_equal(g.density, v["density"])
    np.testing.assert_array_equal(g.color, v["color"])
    ref.close()
