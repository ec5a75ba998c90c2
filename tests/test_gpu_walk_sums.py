"""The leaf walk's sums and classification where they leave their fast forms:
colours below 0 and above 1 (signed 64-bit terms), exactly 0 and 1, opaque
Gaussians (terms of a whole unit), many Gaussians on one voxel (carries into the
high words), boxes one voxel thin and as wide as a leaf, clouds far from the
origin (the reference test on most voxels).  Bit-exact against the oracle."""

import numpy as np
import pytest

from nanovdb_editor import workloads as W

pytestmark = pytest.mark.gpu

NAMES = ("means", "quats", "scales", "opacities", "colors")


def _cloud(kind, n, vs, seed):
    rng = np.random.default_rng(seed)
    c = W.plain_cloud(n, seed)
    c["means"] = rng.uniform(-12 * vs, 12 * vs, (n, 3)).astype(np.float32)
    c["scales"] = (vs * np.exp(rng.normal(np.log(1.0), 0.5, (n, 3)))).astype(np.float32)
    if kind == "colors":
        c["colors"] = rng.uniform(-2.0, 3.0, (n, 3)).astype(np.float32)
        c["colors"][::3] = rng.integers(0, 2, c["colors"][::3].shape)
    elif kind == "opaque":
        c["opacities"][:] = 1.0
        c["colors"][:] = 1.0
        c["scales"] *= 4
    elif kind == "stack":
        c["means"][:] = (0.3 * vs, -0.2 * vs, 0.1 * vs)
        c["opacities"][:] = rng.uniform(0.02, 1.0, n)
    elif kind == "thin":
        c["quats"][:] = (1, 0, 0, 0)
        c["scales"] = (vs * rng.choice([0.01, 0.13, 3.0, 6.0], (n, 3))).astype(np.float32)
    elif kind == "far":
        c["means"] += np.array([30000 * vs, -29000 * vs, 1000 * vs], np.float32)
    return c


@pytest.mark.parametrize("kind", ["colors", "opaque", "stack", "thin", "far"])
@pytest.mark.parametrize("n,vs", [(13, 0.01), (700, 0.004)])
def test_walk_matches_oracle(vox_ctx, oracle_mod, kind, n, vs):
    c = _cloud(kind, n, vs, n)
    g = vox_ctx.voxelize_host(*[c[k] for k in NAMES], vs, 100.0)
    ref = oracle_mod.OracleResult(c, vs, 100.0, window_mode=0)
    assert g.counts["pairs"] == ref.counts["P"] and g.counts["voxels"] == ref.counts["V"]
    assert np.array_equal(g.node2, ref.node2())
    v = ref.values()
    for k in ("rgba8", "density", "color"):
        np.testing.assert_array_equal(getattr(g, k), v[k])
    k_ref, i_ref = ref.pairs()
    k_got, i_got = vox_ctx.pairs()
    np.testing.assert_array_equal(k_got, k_ref)
    np.testing.assert_array_equal(i_got, i_ref)
    ref.close()


@pytest.mark.parametrize("check", [False, True])
@pytest.mark.parametrize("kind", ["colors", "opaque", "stack", "thin", "far"])
def test_differentiable_walk_keeps_the_bytes(oracle_mod, monkeypatch, kind, check):
    """The differentiable channels' walk decides the RGBA8 alpha from its own, approximate
    evaluation; the bytes are the oracle's.  check: every decided byte against the
    reference's evaluation on the device."""
    from nanovdb_editor.vox import FLAG_DIFFERENTIABLE, VoxContext

    if check:
        monkeypatch.setenv("VOX_CHECK_EMIT", "1")
    ctx = VoxContext(0)
    for n, vs in ((13, 0.01), (700, 0.004)):
        c = _cloud(kind, n, vs, n + 1)
        g = ctx.voxelize_host(*[c[k] for k in NAMES], vs, 100.0, FLAG_DIFFERENTIABLE)
        ref = oracle_mod.OracleResult(c, vs, 100.0, window_mode=0)
        np.testing.assert_array_equal(g.rgba8, ref.values()["rgba8"])
        ref.close()
    ctx.close()
