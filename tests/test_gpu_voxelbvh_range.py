"""VoxelBVH ingestion where the certified cell test's numbers near the end of float32's
range (worlds down to 1e-36, cells of 2^-127): the bits of the oracle's cells."""

import numpy as np
import pytest

from nanovdb_editor import workloads as W
from test_gpu_voxelbvh import _compare, _run, _transform

pytestmark = pytest.mark.gpu

RES = 256


def _cloud(unit):
    """A cloud in a box of about 1, in units of 2^-unit: the cells are 2^-(unit + 8)."""
    c = W.plain_cloud(700, 77)
    rng = np.random.default_rng(unit)
    c["means"] = rng.uniform(-0.5, 0.5, (700, 3))
    c["scales"] = 0.01 * np.exp(rng.uniform(-1, 1, (700, 3)))
    for k in ("means", "scales"):
        c[k] = np.ldexp(c[k], -unit).astype(np.float32)
    return c


@pytest.mark.parametrize("unit", [0, 80, 110, 117, 118, 119])
def test_small_worlds(vox_ctx, oracle_mod, unit):
    c = _cloud(unit)
    _compare(_run(vox_ctx, c, RES), oracle_mod.voxelbvh_ijkl(c, RES))


@pytest.mark.parametrize("unit", [0, 80, 110, 118, 119])
def test_small_worlds_under_a_transform(vox_ctx, oracle_mod, unit):
    c = _cloud(unit)
    T = _transform()
    T[3, :3] = 0.0
    Ti = vox_ctx.voxelbvh_transform_inverse(T)
    _compare(_run(vox_ctx, c, RES, T), oracle_mod.voxelbvh_ijkl(c, RES, T, Ti))
