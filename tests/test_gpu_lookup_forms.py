"""The target lookup's splitter table at its own edges (key counts around multiples of the
part size, parts past the last key), and callers that have to see torch's operators:
function modes, vmap, make_fx, tensors whose memory is not their value."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _grid(keys, density, device="cuda"):
    import torch

    from nanovdb_editor.autograd import BatchTargetGrid

    g = BatchTargetGrid(keys, torch.ones(keys.shape, dtype=torch.bool), density)
    g.keys, g.density = g.keys.to(device), g.density.to(device)
    return g


# 256 queries per block: 256 parts where there are 512 keys or more, of 2, 3, 4 keys
@pytest.mark.parametrize("count", [255, 256, 257, 511, 512, 513, 514, 767, 768, 769, 1023, 1024, 1025])
def test_splitter_edges(vox_ctx, count):
    import torch

    from nanovdb_editor.autograd import _fused_lookup

    k = np.sort(np.random.default_rng(count).choice(1 << 40, count, replace=False)) * 2
    keys, dens = torch.from_numpy(k), torch.arange(1.0, count + 1.0)
    far = np.array([-(1 << 63), -1, 0, (1 << 63) - 1], np.int64)
    q = np.concatenate([k, k - 1, k + 1, far])
    q = torch.from_numpy(np.resize(np.random.default_rng(1).permutation(q), (q.size + 255) // 256 * 256))
    dev = _grid(keys, dens)
    assert _fused_lookup(dev.keys, dev.density, None, q.cuda(), False) is not None
    assert torch.equal(dev.lookup(q.cuda()).cpu(), _grid(keys, dens, "cpu").lookup(q))


def test_callers_that_see_the_operators(vox_ctx):
    import torch
    from torch.fx.experimental.proxy_tensor import make_fx
    from torch.overrides import TorchFunctionMode

    from nanovdb_editor.autograd import _fused_lookup

    keys = torch.arange(0, 3000, 3)
    g = _grid(keys, torch.arange(1000.0))
    q = torch.arange(-10, 3010, device="cuda")
    want = g.lookup(q)

    class Names(TorchFunctionMode):
        def __init__(self):
            super().__init__()
            self.seen = []

        def __torch_function__(self, func, types, args=(), kwargs=None):
            self.seen.append(getattr(func, "__name__", str(func)))
            return func(*args, **(kwargs or {}))

    with Names() as mode:
        got = g.lookup(q)
    assert "searchsorted" in mode.seen and torch.equal(got, want)
    graph = make_fx(lambda x: g.lookup(x))(q)
    assert "searchsorted" in graph.code and torch.equal(graph(q), want)
    rows = torch.stack([q, q + 3])
    assert torch.equal(torch.vmap(g.lookup)(rows), torch.stack([want, g.lookup(q + 3)]))
    with torch.device("cuda"):  # a default device is no reason
        assert _fused_lookup(g.keys, g.density, None, q, False) is not None


def test_tensors_without_their_values_in_memory(vox_ctx):
    import torch

    from nanovdb_editor.autograd import _fused_lookup

    g = _grid(torch.arange(0, 3000, 3), torch.arange(1000.0))
    q = torch.arange(-10, 3010, device="cuda")
    want = g.lookup(q)
    g.density = torch._neg_view(g.density)
    assert torch.equal(g.lookup(q), -want)
    g.density = torch._efficientzerotensor(1000, device="cuda")  # no memory at all
    assert _fused_lookup(g.keys, g.density, None, q, False) is None
