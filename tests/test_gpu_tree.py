"""The tree stage at the edges of its tiles (128 candidate leaves per warp, 1024
per CTA): clouds of one small Gaussian per leaf, some of them on leaf faces (more
candidates than Gaussians, some empty), spread over lower and upper nodes, and
batches with clouds that have no voxel.  Bit-exact against the oracle."""

import numpy as np
import pytest

from nanovdb_editor import workloads as W

pytestmark = pytest.mark.gpu

NAMES = ("means", "quats", "scales", "opacities", "colors")
VS = 0.01


def _lattice_cloud(n, stride, seed):
    """One Gaussian of about a voxel in each of n leaves, `stride` leaves apart."""
    rng = np.random.default_rng(seed)
    side = int(np.ceil(n ** (1.0 / 3.0)))
    at = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    at = (at - side // 2) * 8 * stride
    offset = rng.uniform(2.0, 6.0, (n, 3))
    face = rng.random(n) < 0.2
    offset[face, 0] = rng.uniform(-0.7, 0.7, int(face.sum()))
    c = W.plain_cloud(max(n, 1), seed)
    for k in NAMES:
        c[k] = c[k][:n]
    c["means"] = ((at + offset) * VS).astype(np.float32)
    c["scales"] = rng.uniform(0.1 * VS, 0.4 * VS, (n, 3)).astype(np.float32)
    return c


def _same(g, cloud, oracle_mod):
    ref = oracle_mod.OracleResult(cloud, VS, 0.05, window_mode=0)
    c = ref.counts
    assert (g.counts["upper"], g.counts["lower"], g.counts["leaf"]) == (c["upper"], c["lower"], c["leaf"])
    assert g.counts["pairs"] == c["P"] and g.counts["voxels"] == c["V"]
    assert np.array_equal(g.node2, ref.node2())
    v = ref.values()
    for k in ("rgba8", "density", "color"):
        np.testing.assert_array_equal(getattr(g, k), v[k])
    if c["V"]:
        np.testing.assert_array_equal(g.bbox, ref.bbox())
    ref.close()


@pytest.mark.parametrize("n,stride", [(1, 1), (32, 1), (33, 20), (127, 1), (128, 3), (129, 1), (1023, 1), (1024, 2),
                                      (1025, 17), (5000, 1), (3000, 40)])
def test_tree_matches_oracle(vox_ctx, oracle_mod, n, stride):
    c = _lattice_cloud(n, stride, n)
    _same(vox_ctx.voxelize_host(*[c[k] for k in NAMES], VS), c, oracle_mod)


def test_tree_of_batches_with_empty_clouds(vox_ctx, oracle_mod):
    import torch

    sizes = [0, 5, 0, 0, 130, 1, 0, 1200, 64, 0]
    clouds = [_lattice_cloud(n, 1 + i % 4 * 9, 50 + i) for i, n in enumerate(sizes)]
    start = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (W.concat(clouds)[k] for k in NAMES)]
    torch.cuda.synchronize()
    _, goff, _ = vox_ctx.voxelize_batch(*dev, start, np.full(len(sizes), VS, np.float32))
    for g, c in zip(vox_ctx.grids(goff), clouds):
        _same(g, c, oracle_mod)
