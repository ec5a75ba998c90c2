"""The one-pass target lookup against the same lookup by torch's operators on the
CPU, exactly: key counts around the search's 17-way rounds, query counts around a
warp and a block, equal keys, queries in and out of order, out of the 21-bit
range, and every form that has to stay with the operators."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _coords(rng, n, span):
    return rng.integers(-span, span + 1, (n, 3)).astype(np.int32)


@pytest.mark.parametrize("keys", [0, 1, 2, 15, 16, 17, 18, 288, 289, 290, 4913, 70001])
@pytest.mark.parametrize("n", [0, 1, 31, 33, 257, 20000])
def test_lookup(vox_ctx, keys, n):
    import torch

    from nanovdb_editor.autograd import BatchTargetGrid, TargetGrid, _fused_lookup, pack_coords

    rng = np.random.default_rng(keys * 31 + n)
    span = max(1, round(keys ** (1 / 3) / 1.6))  # dense enough for hits, duplicates included
    target = torch.from_numpy(_coords(rng, keys, span)) + torch.tensor([5, -70000, 300], dtype=torch.int32)
    dens = torch.from_numpy(rng.normal(size=keys).astype(np.float32))
    q = _coords(rng, n, span + 1)
    q[n // 2 :] = q[n // 2 :][np.lexsort(q[n // 2 :].T[::-1])]
    q = torch.from_numpy(q) + torch.tensor([5, -70000, 300], dtype=torch.int32)
    if n > 4:
        q[0] = -(1 << 31)
        q[1] = (1 << 31) - 1
    host = TargetGrid(target, dens)
    dev = TargetGrid(target, dens)
    dev.keys, dev.density = host.keys.cuda(), host.density.cuda()
    want, want_hit = host.lookup(q)
    assert _fused_lookup(dev.keys, dev.density, q.cuda(), None, True) is not None
    got, got_hit = dev.lookup(q.cuda())
    assert torch.equal(got.cpu(), want) and torch.equal(got_hit.cpu(), want_hit)
    # the key form
    bh = BatchTargetGrid(pack_coords(target), torch.ones(keys, dtype=torch.bool), dens)
    bd = BatchTargetGrid(pack_coords(target), torch.ones(keys, dtype=torch.bool), dens)
    bd.keys, bd.density = bh.keys.cuda(), bh.density.cuda()
    assert torch.equal(bd.lookup(pack_coords(q).cuda()).cpu(), bh.lookup(pack_coords(q)))


def test_lookup_with_every_splitter(vox_ctx):
    """Enough queries per block for the largest splitter table, more of them than threads."""
    import torch

    from nanovdb_editor.autograd import BatchTargetGrid

    rng = np.random.default_rng(11)
    keys = torch.from_numpy(rng.integers(0, 300_000, 100_003))
    host = BatchTargetGrid(keys, torch.ones(keys.shape, dtype=torch.bool), torch.from_numpy(rng.normal(size=100_003).astype(np.float32)))
    q = torch.from_numpy(rng.integers(-5, 300_005, 3_000_001))
    dev = BatchTargetGrid(keys, torch.ones(keys.shape, dtype=torch.bool), host.density)
    dev.keys, dev.density = host.keys.cuda(), host.density.cuda()
    assert torch.equal(dev.lookup(q.cuda()).cpu(), host.lookup(q))


def test_forms_left_to_the_operators(vox_ctx):
    import torch

    from nanovdb_editor.autograd import TargetGrid, _fused_lookup

    rng = np.random.default_rng(3)
    c = torch.from_numpy(_coords(rng, 500, 5)).cuda()
    t = TargetGrid(c, torch.arange(500.0, device="cuda"))
    want, hit = t.lookup(c)
    assert bool(hit.all())
    wide = torch.zeros(500, 4, dtype=torch.int32, device="cuda")
    wide[:, :3] = c
    for form in (wide[:, :3], c.long(), c.t().contiguous().t()):
        assert _fused_lookup(t.keys, t.density, form, None, True) is None
        got, h = t.lookup(form)
        assert torch.equal(got, want) and torch.equal(h, hit)
    t.density.requires_grad_(True)
    assert _fused_lookup(t.keys, t.density, c, None, True) is None
    t.lookup(c)[0].sum().backward()
    assert float(t.density.grad.sum()) == 500.0
    t.density = t.density.detach()
    with torch.autograd.forward_ad.dual_level():
        t.density = torch.autograd.forward_ad.make_dual(t.density, torch.ones_like(t.density))
        tangent = torch.autograd.forward_ad.unpack_dual(t.lookup(c)[0]).tangent
        assert torch.equal(tangent, torch.ones(500, device="cuda"))
