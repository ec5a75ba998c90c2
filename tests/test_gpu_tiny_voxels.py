"""Voxel sizes below 1e-22, where the squared scales underflow and the opacity
transform's exponent is infinite: an alpha of 1, or of 0 where 1 - a rounds to 1 (a
lattice point far from a faint Gaussian smaller than a voxel).  Density, colour and RGBA8 against the oracle, bit for bit, and the RGBA8 values of the
differentiable walk and of the entry that returns nothing else."""

import numpy as np
import pytest

from nanovdb_editor import workloads as W

pytestmark = pytest.mark.gpu

NAMES = ("means", "quats", "scales", "opacities", "colors")


def _cloud(n, vs, seed):
    rng = np.random.default_rng(seed)
    c = W.plain_cloud(n, seed)
    c["means"] = (vs * rng.uniform(-12, 12, (n, 3))).astype(np.float32)
    c["scales"] = (vs * np.exp(rng.uniform(np.log(0.02), np.log(4.0), (n, 3)))).astype(np.float32)
    c["scales"][::2] = 0.02 * vs
    c["opacities"] = np.exp(rng.uniform(np.log(0.0101), 0.0, n)).astype(np.float32)
    return c


@pytest.mark.parametrize("vs", [1e-18, 3e-21, 1e-22, 4e-23, 1e-23, 1e-25, 1e-30, 1e-36])
@pytest.mark.parametrize("n", [1, 40, 700])
def test_every_channel(vox_ctx, oracle_mod, n, vs):
    from nanovdb_editor import Compute, Raster
    from nanovdb_editor.grid import NodeGrid
    from nanovdb_editor.vox import FLAG_DIFFERENTIABLE

    vs = float(np.float32(vs))
    c = _cloud(n, vs, n + 5)
    ref = oracle_mod.OracleResult(c, vs, 0.05, window_mode=0)
    assert ref.counts["error"] == 0 and ref.counts["V"] > 0
    v = ref.values()
    g = vox_ctx.voxelize_host(*[c[k] for k in NAMES], vs, 0.05)
    np.testing.assert_array_equal(g.node2, ref.node2())
    np.testing.assert_array_equal(g.rgba8, v["rgba8"])
    np.testing.assert_array_equal(g.density, v["density"])
    np.testing.assert_array_equal(g.color, v["color"])
    smooth = vox_ctx.voxelize_host(*[c[k] for k in NAMES], vs, 0.05, flags=FLAG_DIFFERENTIABLE)
    np.testing.assert_array_equal(smooth.rgba8, v["rgba8"])
    compute = Compute(device_index=0)
    raster = Raster(compute)
    arrs = {k: compute.create_array(np.ascontiguousarray(c[k])) for k in ("means", "quats", "scales", "colors", "opacities")}
    sh0, shn = (compute.create_array(np.zeros(0, np.float32)) for _ in range(2))
    out = raster.raster_to_nanovdb(vs, arrs["means"], arrs["quats"], arrs["scales"], arrs["colors"], sh0, shn, arrs["opacities"])
    only = NodeGrid(np.array(compute.map_array(out, np.uint8)))
    np.testing.assert_array_equal(only.rgba8, v["rgba8"])
    for a in [*arrs.values(), sh0, shn, out]:
        compute.destroy_array(a)
    ref.close()
