"""Timing cases of the Gaussian -> NanoVDB framework: what a user's program asks of it, from the
32-Gaussian cloud of a pipeline test to the 2M-Gaussian scene, each through the public entry points.

Kinds of case
  forward   VoxContext.voxelize of device tensors, the grid taken over as a torch tensor
  host      Raster.raster_to_nanovdb_from_arrays: host arrays in, host grid out (window node order)
  fit       one fitting step: autograd.voxelize, the L2 loss to a target grid, the adjoint
  batch     VoxContext.voxelize_batch of many uneven clouds in one call
  batch_fit one batched fitting step: differentiable forward, L2 per cloud, the adjoint
  bvh       VoxContext.voxelbvh_ijkl_from_gaussians

Every case gives the number of Gaussians `n` (all clouds together for batches), the distribution of
the cloud (`dist`: "plain" fills a cube uniformly, "cluster" lies on `clusters` surface-like sheets)
and the voxel size `vs` (the smallest of a batch).  How many voxels and nodes come of it depends on
the values, so a program keeps buffers of a capacity (`_capacity`) and finds its results at their front.
"""

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "nanovdb-editor_b200"))

from nanovdb_editor import Compute, Raster  # noqa: E402
from nanovdb_editor.autograd import BatchTargetGrid, TargetGrid, l2_to_batch_target, voxelize  # noqa: E402
from nanovdb_editor.grid import HEADER_DTYPE, NodeGrid  # noqa: E402
from nanovdb_editor.vox import FLAG_BF16_INPUTS, FLAG_DIFFERENTIABLE, FLAG_RAW_INPUTS, FLAG_WINDOW_ORDER, VoxContext  # noqa: E402

NAMES = ("means", "quats", "scales", "opacities", "colors")
SH_C0 = 0.28209479177387814
COLOR_WEIGHT = 0.05  # the fitting loss' colour term

# log-scale mean and deviation of the distributions, as nanovdb_editor.workloads draws them
SCALES = {"plain": (0.01, 0.3), "cluster": (0.003, 0.5), "sparse": (0.02, 0.3)}


def _case(name, kind, n, dist, vs, clusters=1, clouds=1, raw=True, bf16=False, window=False, res=0, transform=False):
    return {"name": name, "kind": kind, "n": n, "dist": dist, "vs": vs, "clusters": clusters, "clouds": clouds,
            "raw": raw, "bf16": bf16, "window": window, "res": res, "transform": transform}


def listed():
    return [
        # a cloud of the pipeline test's size: an interactive edit of a handful of splats, all latency
        _case("forward_32", "forward", 32, "sparse", 0.05),
        # a small ragged cloud of activated attributes, nodes in the reference's window order
        _case("forward_4999_window", "forward", 4999, "plain", 0.01, raw=False, window=True),
        # the reference's CPU-sized workload: 100k Gaussians filling a cube
        _case("forward_100k", "forward", 100_000, "plain", 0.01),
        # the at-scale scene
        _case("forward_2M", "forward", 2_000_000, "cluster", 0.002, clusters=64),
        # the drop-in table entry on host arrays, at the size of one object and of a room
        _case("host_30k", "host", 30_011, "plain", 0.01),
        _case("host_500k", "host", 500_000, "cluster", 0.004, clusters=64),
        # fitting steps: a small scene, and the 500k-Gaussian fit
        _case("fit_20k", "fit", 20_003, "plain", 0.015),
        _case("fit_500k", "fit", 500_000, "cluster", 0.004, clusters=64),
        # many uneven clouds in one call: a data-set conversion, and a batched bfloat16 fit
        _case("batch_64", "batch", 2_000_000, "cluster", 0.002, clouds=64),
        _case("batch_fit_16_bf16", "batch_fit", 600_000, "cluster", 0.004, clouds=16, bf16=True),
        # ingestion of the same splats into the VoxelBVH builder's keys
        _case("bvh_20k_transform", "bvh", 20_011, "plain", 0.01, res=256, transform=True),
        _case("bvh_2M", "bvh", 2_000_000, "cluster", 0.002, clusters=64, res=512),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["forward", "forward", "forward", "host", "fit", "fit", "batch", "batch_fit", "bvh", "bvh"])
    dist = rng.choice(["plain", "cluster"])
    most = {"forward": 2_000_000, "host": 500_000, "fit": 500_000, "batch": 2_000_000, "batch_fit": 600_000,
            "bvh": 2_000_000}[kind]
    n = int(_log_uniform(rng, 32, most)) | 1
    clouds = 1
    if kind.startswith("batch"):
        dist = "cluster"
        n = max(n, 64)
        clouds = rng.randint(2, 64 if kind == "batch" else 16)
    vs = _log_uniform(rng, 0.008, 0.03) if dist == "plain" else _log_uniform(rng, 0.002, 0.02)
    c = _case("", kind, n, dist, vs, clusters=rng.randint(1, 64), clouds=clouds, raw=rng.random() < 0.7,
              bf16=kind in ("forward", "fit", "batch_fit") and rng.random() < 0.3,
              window=kind == "forward" and rng.random() < 0.3, res=0, transform=False)
    if kind in ("host", "batch_fit"):
        c["raw"] = True
    if kind == "bvh":
        c["res"] = int(_log_uniform(rng, 32, 4096))
        c["transform"] = rng.random() < 0.3
    if kind == "forward":  # a larger voxel where the scene would outgrow the largest listed one
        while _pairs(c) > 1.2e9:
            c["vs"] *= 1.2
    elif kind != "bvh":
        while _pairs(c) > 3e8:
            c["vs"] *= 1.2
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs ----
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _cloud(n, dist, clusters, seed):
    """Activated attributes of one cloud (the distributions of nanovdb_editor.workloads)."""
    g = _generator(seed)

    def uniform(lo, hi, *shape):
        return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo

    def normal(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)

    mean, sigma = SCALES[dist]
    if dist == "sparse":
        means = 0.3 * normal(n, 3)
    elif dist == "plain":
        means = uniform(-1.0, 1.0, n, 3)
    else:
        centre = uniform(-1.0, 1.0, clusters, 3)
        frame = torch.linalg.qr(normal(clusters, 3, 3))[0]
        cid = torch.randint(0, clusters, (n,), generator=g, device="cuda")
        local = normal(n, 3) * torch.tensor([0.1, 0.1, 0.005], device="cuda", dtype=torch.float64)
        means = centre[cid] + (frame[cid] @ local[:, :, None])[:, :, 0]
    scales = torch.exp(math.log(mean) + sigma * normal(n, 3))
    scales = torch.maximum(scales, scales.amax(dim=1, keepdim=True) / 20.0)
    quats = normal(n, 4)
    quats /= quats.norm(dim=1, keepdim=True)
    opac = uniform(0.05, 1.0, n)
    colors = uniform(0.0, 1.0, n, 3)
    out = dict(zip(NAMES, (means, quats, scales, opac, colors)))
    return {k: v.to(torch.float32) for k, v in out.items()}


def _raw(c):
    """Log scales, opacity logits, SH0 colours (the on-disk convention)."""
    op = c["opacities"].double().clamp(1e-7, 1.0 - 1e-7)
    return {"means": c["means"], "quats": c["quats"], "scales": c["scales"].double().log().float(),
            "opacities": (op / (1.0 - op)).log().float(), "colors": ((c["colors"].double() - 0.5) / SH_C0).float()}


def _batch_layout(case):
    """Cloud sizes, cluster counts and voxel sizes of a batch: the case's alone, not the seed's."""
    rng = np.random.default_rng(case["n"] * 1009 + case["clouds"])
    B = case["clouds"]
    w = np.exp(rng.uniform(0.0, math.log(200.0), B))
    sizes = np.maximum(1, (w / w.sum() * case["n"]).astype(np.int64))
    start = np.zeros(B + 1, dtype=np.int64)
    start[1:] = np.cumsum(sizes)
    clusters = rng.integers(1, 17, B)
    vs = (case["vs"] * np.exp(rng.uniform(0.0, math.log(10.0 if case["kind"] == "batch" else 3.0), B))).astype(np.float32)
    return start, clusters, vs


def _inputs(case, seed):
    if case["clouds"] > 1:
        start, clusters, _ = _batch_layout(case)
        parts = [_cloud(int(b - a), case["dist"], int(k), int(seed) * 1000 + i)
                 for i, (a, b, k) in enumerate(zip(start[:-1], start[1:], clusters))]
        c = {k: torch.cat([p[k] for p in parts]).contiguous() for k in NAMES}
    else:
        c = _cloud(case["n"], case["dist"], case["clusters"], int(seed) * 1000)
    if case["raw"]:
        c = _raw(c)
    return {k: (v.to(torch.bfloat16) if case["bf16"] else v).contiguous() for k, v in c.items()}


def _transform():
    a, b = 0.4, -0.7
    rx = np.array([[1, 0, 0], [0, math.cos(a), -math.sin(a)], [0, math.sin(a), math.cos(a)]])
    rz = np.array([[math.cos(b), -math.sin(b), 0], [math.sin(b), math.cos(b), 0], [0, 0, 1]])
    m = np.eye(4)
    m[:3, :3] = 1.5 * rx @ rz
    m[3, :3] = (0.25, -0.5, 0.125)
    return m.astype(np.float32)


# --------------------------------------------------------------- the program ----
_program = {}


def _context():
    """The program's one voxelization context; it lives as long as the program."""
    if "context" not in _program:
        _program["context"] = VoxContext(0)
    return _program["context"]


def _raster():
    if "raster" not in _program:
        _program["compute"] = Compute()
        _program["raster"] = Raster(_program["compute"])
    return _program["compute"], _program["raster"]


def _flags(case):
    return ((FLAG_RAW_INPUTS if case["raw"] else 0) | (FLAG_BF16_INPUTS if case["bf16"] else 0) |
            (FLAG_WINDOW_ORDER if case["window"] else 0))


class _HostArrays:
    """The library's input arrays, given back when the program drops them."""

    def __init__(self, compute, arrays):
        self.compute = compute
        self.arrays = [compute.create_array(a) for a in arrays]

    def __del__(self):
        for a in self.arrays:
            self.compute.destroy_array(a)


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    t = _inputs(case, seed)
    if kind == "host":
        compute, _ = _raster()
        order = ("means", "opacities", "quats", "scales", "colors")
        state["host"] = _HostArrays(compute, [t[k].cpu().numpy() for k in order] + [np.zeros(0, np.float32)])
        state["grid"] = torch.zeros(_capacity(case)[0], dtype=torch.uint8)
        return state
    state["in"] = [t[k] for k in NAMES]
    ctx = _context()
    if kind != "bvh":
        grid_bytes, voxels = _capacity(case)
        state["grid"] = torch.zeros(grid_bytes, dtype=torch.uint8, device="cuda")
        if kind != "batch":
            state["density"] = torch.zeros(voxels, dtype=torch.float32, device="cuda")
        if kind == "fit":
            state["color"] = torch.zeros(voxels, 3, dtype=torch.float32, device="cuda")
    if kind == "fit":  # the target: the grid of an independently drawn cloud
        other = _inputs(case, int(seed) + 500_009)
        with torch.no_grad():
            density, _, _ = voxelize(*[other[k] for k in NAMES], case["vs"], raw=case["raw"], context=ctx)
        state["target"] = TargetGrid(_coords(ctx, density.shape[0])[2:], density[2:])
        for p in state["in"]:
            p.requires_grad_(True)
    elif kind in ("batch", "batch_fit"):
        state["start"], _, state["vs"] = _batch_layout(case)
        if kind == "batch_fit":
            other = _inputs(case, int(seed) + 500_009)
            torch.cuda.synchronize()
            _, goff, voff = ctx.voxelize_batch(*[other[k] for k in NAMES], state["start"], state["vs"], 0.05,
                                               _flags(case) | FLAG_DIFFERENTIABLE)
            keys, valid = _batch_keys(ctx, voff)
            state["target"] = BatchTargetGrid(keys, valid, _batch_density(ctx, goff, state["grid"]))
            state["grads"] = {k: torch.empty(p.shape, dtype=torch.float32, device="cuda")
                              for k, p in zip(NAMES, state["in"])}
    elif kind == "bvh":
        state["transform"] = _transform() if case["transform"] else None
        if case["raw"]:  # this entry takes activated attributes
            c = _cloud(case["n"], case["dist"], case["clusters"], int(seed) * 1000)
            state["in"] = [c[k] for k in NAMES]
    torch.cuda.synchronize()  # the library reads on a stream of its own
    return state


def _density(grid):
    """The density channel of a grid, as a view of it."""
    h = np.frombuffer(grid[:256].cpu().numpy().tobytes(), HEADER_DTYPE)[0]
    off, voxels = int(h["density_offset"]), int(h["value_count"])
    return grid[off: off + 4 * voxels].view(torch.float32)


def _batch_density(ctx, goff, grid):
    """Every cloud's density of the last batched grid, clouds back to back; the grid is copied to `grid`."""
    torch.cuda.current_stream().synchronize()  # the library writes on its own stream
    ctx.grid_device(grid)
    heads = torch.stack([grid[int(o): int(o) + 256] for o in goff[:-1]]).cpu().numpy().tobytes()
    return torch.cat([grid[int(o) + int(h["density_offset"]): int(o) + int(h["density_offset"]) + 4 * int(h["value_count"])]
                      for o, h in zip(goff[:-1], np.frombuffer(heads, HEADER_DTYPE))]).view(torch.float32)


def _coords(ctx, count):
    """(i, j, k) of every value index of the last grid (the background slots' rows are not set)."""
    coords = torch.empty(count, 3, dtype=torch.int32, device="cuda")
    torch.cuda.current_stream().synchronize()  # the library writes on its own stream
    ctx.voxel_coords(coords)
    return coords


def _batch_keys(ctx, voff):
    """(cloud, i, j, k) of every value index of the last batched grid as one integer, and which are voxels."""
    coords = _coords(ctx, int(voff[-1])).to(torch.int64)
    voff = torch.from_numpy(voff.astype(np.int64)).cuda()
    counts = voff[1:] - voff[:-1]
    cloud = torch.repeat_interleave(torch.arange(counts.numel(), device="cuda"), counts)
    valid = torch.arange(cloud.numel(), device="cuda") - voff[cloud] >= 2
    return torch.where(valid, (cloud << 54) | _key(coords), torch.full_like(cloud, -1)), valid


def _front(buffer, values):
    buffer[: values.shape[0]].copy_(values)
    return buffer


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "host":
        compute, raster = _raster()
        host = state["host"]
        result = raster.raster_to_nanovdb_from_arrays(case["vs"], host.arrays)
        _front(state["grid"], torch.from_numpy(compute.map_array(result, np.uint8)))
        compute.destroy_array(result)
        return state["grid"]
    ctx = _context()
    if kind == "forward":
        ctx.voxelize(*state["in"], case["vs"], 0.05, _flags(case))
        ctx.grid_device(state["grid"])
        return {"grid": state["grid"], "density": _front(state["density"], _density(state["grid"]))}
    if kind == "fit":
        density, color, grid = voxelize(*state["in"], case["vs"], raw=case["raw"], context=ctx)
        want, _ = state["target"].lookup(_coords(ctx, density.shape[0])[2:])
        loss = 0.5 * ((density[2:] - want) ** 2).sum() + COLOR_WEIGHT * (color ** 2).sum()
        grads = torch.autograd.grad(loss, state["in"])
        with torch.no_grad():
            return {"loss": loss.detach(), "density": _front(state["density"], density),
                    "color": _front(state["color"], color), "grads": dict(zip(NAMES, grads))}
    if kind == "batch":
        _, goff, voff = ctx.voxelize_batch(*state["in"], state["start"], state["vs"], 0.05, _flags(case))
        ctx.grid_device(state["grid"])
        return {"grid": state["grid"], "grid_offsets": goff.astype(np.int64), "value_offsets": voff.astype(np.int64)}
    if kind == "batch_fit":
        _, goff, voff = ctx.voxelize_batch(*state["in"], state["start"], state["vs"], 0.05,
                                           _flags(case) | FLAG_DIFFERENTIABLE)
        density = _batch_density(ctx, goff, state["grid"])
        keys, valid = _batch_keys(ctx, voff)
        loss, gd = l2_to_batch_target(density, keys, valid, state["target"])
        gd = gd.contiguous()
        torch.cuda.current_stream().synchronize()  # the adjoint reads gd on the library's stream
        ctx.backward(*state["in"], gd, None, state["grads"])
        return {"loss": loss, "density": _front(state["density"], density), "grads": state["grads"]}
    means, quats, scales, opacities, _ = state["in"]
    return ctx.voxelbvh_ijkl_from_gaussians(means, opacities, quats, scales, case["res"], state["transform"])


# ---------------------------------------------------------------------- work ----
def _pairs_at(n, dist, vs):
    """(voxel, Gaussian) pairs: the 0.01-opacity ellipsoid, grown by a little over a voxel."""
    mean, sigma = SCALES[dist]
    r = 2.7 * mean * math.exp(0.5 * sigma * sigma) / vs + 1.15
    return n * 4.0 / 3.0 * math.pi * r ** 3


def _voxels_at(n, dist, vs, clusters):
    """Active voxels: the pairs spread over the volume the cloud fills."""
    space = {"plain": 8.0, "cluster": 0.0135 * clusters, "sparse": 2.0}[dist] / vs ** 3
    return space * -math.expm1(-_pairs_at(n, dist, vs) / space)


def _parts(case):
    if case["clouds"] == 1:
        return [(case["n"], case["vs"], case["clusters"])]
    start, clusters, vs = _batch_layout(case)
    return [(int(b - a), float(v), int(k)) for a, b, v, k in zip(start[:-1], start[1:], vs, clusters)]


def _pairs(case):
    return sum(_pairs_at(n, case["dist"], vs) for n, vs, _ in _parts(case))


def _capacity(case):
    """Bytes and value slots that hold the case's grids whatever the seed."""
    nbytes, values = 4096, 0
    for n, vs, clusters in _parts(case):
        mean, sigma = SCALES[case["dist"]]
        reach = 2.7 * mean * math.exp(0.5 * sigma * sigma) / vs
        space = {"plain": 8.0, "cluster": 0.0135 * clusters, "sparse": 2.0}[case["dist"]] / vs ** 3
        voxels = int(1.4 * _voxels_at(n, case["dist"], vs, clusters)) + 4 * n + 1000
        leaves = int(min(voxels, n * (reach / 4 + 2) ** 3, 6 * space / 512 + 4 * n)) + 100
        lowers = int(min(leaves, (4.0 / (128 * vs) + 2) ** 3, 16 * n))
        uppers = int(min(lowers, (4.0 / (4096 * vs) + 2) ** 3))
        nbytes += 541728 + 8192 + uppers * 274464 + lowers * 34336 + leaves * 128 + 20 * voxels
        values += voxels + 2
    return nbytes, values


def work(case):
    """Inputs read once, outputs written once; per pair the ellipsoid test, the alpha and the sums (about
    100 operations; the adjoint's 19 terms about as many again)."""
    n, kind = case["n"], case["kind"]
    if kind == "bvh":  # 8 keys, ids and headers per Gaussian; about ten cells tested, 60 operations each
        return {"bytes": 44 * n + n * (8 * 8 + 8 * 4 + 16 * 4) + 24, "flops": 600 * n}
    inputs = (28 if case["bf16"] else 56) * n
    voxels = sum(_voxels_at(m, case["dist"], vs, k) for m, vs, k in _parts(case))
    pairs = _pairs(case)
    nodes = 541728 * case["clouds"] + voxels * (128 / 277.0 + 0.2)
    grid = nodes + voxels * (4 if kind == "host" else 20)
    if kind in ("fit", "batch_fit"):  # gradients of the channels read, of the attributes written
        return {"bytes": 2 * inputs + 56 * n + grid + 16 * voxels, "flops": 200 * pairs}
    return {"bytes": inputs + grid, "flops": 100 * pairs}


# ------------------------------------------------------------- 64-bit answers ----
def _activated64(t, raw):
    """means, unit quaternions, scales, opacities, colours in 64 bits."""
    mu, q, s, op, col = (t[k].double() for k in NAMES)
    if raw:
        q = q / q.norm(dim=1, keepdim=True)
        s, op, col = torch.exp(s), torch.sigmoid(op), SH_C0 * col + 0.5
    return mu, q, s, op, col


def _rotation(q):
    w, x, y, z = q.unbind(1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                        2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                        2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], 1).view(-1, 3, 3)


def _boxes(mu, q, s, op, vs):
    """Per Gaussian the voxel box of its 0.01-opacity ellipsoid: (origin, extent), extent 0 where it has none."""
    ls = torch.sqrt(2.0 * torch.log((op / 0.01).clamp(min=1.0)))
    half = (_rotation(q) * (ls[:, None] * s.clamp(min=0.125 * vs))[:, None, :]).abs().sum(2)
    lo, hi = torch.floor((mu - half) / vs), torch.floor((mu + half) / vs)
    ext = torch.where((op > 0.01)[:, None], hi - lo + 1, torch.zeros_like(lo))
    return lo.long(), ext.long(), ls


def _candidates(lo, ext, most=20_000_000):
    """The boxes' voxels in chunks: (Gaussian index, voxel coordinates)."""
    count = ext.prod(1)
    ends = torch.cumsum(count, 0).cpu().numpy()
    a, n = 0, int(count.numel())
    while a < n:
        base = int(ends[a - 1]) if a else 0
        b = max(a + 1, int(np.searchsorted(ends, base + most, side="right")))
        c = count[a:b]
        g = torch.repeat_interleave(torch.arange(a, b, device=c.device), c)
        i = torch.arange(g.numel(), device=c.device) - (torch.cumsum(c, 0) - c)[g - a]
        yz = ext[g, 1] * ext[g, 2]
        ijk = torch.stack([i // yz, (i % yz) // ext[g, 2], i % ext[g, 2]], 1) + lo[g]
        yield g, ijk
        a = b


def _smooth(mu, q, s, op, g, ijk, vs):
    """The differentiable channels' kernel of the pairs (g, ijk)."""
    d = (ijk.double() + 0.5) * vs - mu[g]
    z = (_rotation(q)[g] * d[:, :, None]).sum(1) / s.clamp(min=0.125 * vs)[g]
    return (op[g] * torch.exp(-0.5 * (z * z).sum(1)) - 0.01).clamp(min=0.0)


def _key(ijk):
    b = ijk + (1 << 17)
    return (b[:, 0] << 36) | (b[:, 1] << 18) | b[:, 2]


def _smooth_grid(t, raw, vs):
    """Voxel keys, densities and colour sums of a cloud's differentiable channels."""
    mu, q, s, op, col = _activated64(t, raw)
    lo, ext, _ = _boxes(mu, q, s, op, vs)
    keys, parts = [], []
    for g, ijk in _candidates(lo, ext):
        k = _smooth(mu, q, s, op, g, ijk, vs)
        on = k > 0
        u, inv = torch.unique(_key(ijk[on]), return_inverse=True)
        v = torch.zeros(u.numel(), 4, dtype=torch.float64, device=u.device)
        v.index_add_(0, inv, torch.cat([k[on, None], k[on, None] * col[g[on]]], 1))
        keys.append(u)
        parts.append(v)
    u, inv = torch.unique(torch.cat(keys), return_inverse=True)
    v = torch.zeros(u.numel(), 4, dtype=torch.float64, device=u.device)
    return u, v.index_add_(0, inv, torch.cat(parts))


def _fit_grads(t, other, raw, vs, color_weight):
    """Loss and gradients of 0.5 |density - target|^2 + color_weight |colour|^2 over the cloud's voxels, and
    0.5 |target|^2 over the voxels that only the target has."""
    vs = float(np.float32(vs))
    keys, v = _smooth_grid(t, raw, vs)
    tkeys, tv = _smooth_grid(other, raw, vs)
    pos = torch.searchsorted(tkeys, keys).clamp(max=max(tkeys.numel() - 1, 0))
    hit = tkeys[pos] == keys
    want = torch.where(hit, tv[pos, 0], torch.zeros_like(v[:, 0]))
    err, cgrad = v[:, 0] - want, 2.0 * color_weight * v[:, 1:]
    loss = 0.5 * (err ** 2).sum() + color_weight * (v[:, 1:] ** 2).sum()
    missing = 0.5 * ((tv[:, 0] ** 2).sum() - (want ** 2).sum())
    params = {k: t[k].double().detach().requires_grad_(True) for k in NAMES}
    with torch.no_grad():
        lo, ext, _ = _boxes(*_activated64(params, raw)[:4], vs)
    grads = [torch.zeros_like(p) for p in params.values()]
    for g, ijk in _candidates(lo, ext, 10_000_000):
        mu, q, s, op, col = _activated64(params, raw)
        with torch.no_grad():
            key = _key(ijk)
            at = torch.searchsorted(keys, key).clamp(max=keys.numel() - 1)
            on = keys[at] == key
            g, ijk, at = g[on], ijk[on], at[on]
        k = _smooth(mu, q, s, op, g, ijk, vs)
        part = (k * (err[at] + (cgrad[at] * col[g]).sum(1))).sum()
        for acc, new in zip(grads, torch.autograd.grad(part, list(params.values()))):
            acc += new
    return loss, missing, dict(zip(NAMES, grads))


def _forward_density(t, raw, vs, cull=0.05):
    """Density by value index (canonical node order): every pair whose voxel box reaches the 0.01-opacity
    ellipsoid adds 1 - (1 - op exp(-ls d))^(vs / (0.1 |s|)), d the smallest squared distance of the box's
    4 x 4 x 4 lattice."""
    vs = float(np.float32(vs))
    mu, q, s, op, _ = _activated64(t, raw)
    lo, ext, ls = _boxes(mu, q, s, op, vs)
    s = s.clamp(min=0.125 * vs)
    rot = _rotation(q)
    size = s.norm(dim=1)
    keys, parts = [], []
    for g, ijk in _candidates(lo, ext):
        centre = (ijk.double() + 0.5) * vs - mu[g]
        scale = 1.0 / (ls[:, None] * s)[g]
        mid = (rot[g] * centre[:, :, None]).sum(1) * scale
        half = 0.5 * vs * rot.abs().sum(1)[g] * scale
        a, b = mid - half, mid + half
        near = torch.where(a > 0, a, torch.where(b < 0, b, torch.zeros_like(a)))
        on = (near ** 2).sum(1) < 1.0
        g, ijk, a, b = g[on], ijk[on], a[on], b[on]
        d = torch.stack([(a + w * (b - a)) ** 2 for w in (0.0, 1.0 / 3.0, 2.0 / 3.0, 1.0)]).amin(0).sum(1)
        al = 1.0 - (1.0 - op[g] * torch.exp(-ls[g] * d)) ** (vs / (0.1 * size[g]))
        keys.append(_node_key(ijk))
        parts.append(torch.where(size[g] > cull, torch.zeros_like(al), al))
    u, inv = torch.unique(torch.cat(keys), return_inverse=True)
    return torch.zeros(u.numel() + 2, dtype=torch.float64, device=u.device).index_add_(0, inv + 2, torch.cat(parts))


def _node_key(ijk):
    """Hierarchical key (root tile, upper, lower, leaf slot): ascending keys are canonical value order."""
    x, y, z = (ijk & 0x1FFFF).unbind(1)
    key = torch.zeros_like(x)
    for shift, bits in ((12, 5), (7, 5), (3, 4), (0, 3)):
        m = (1 << bits) - 1
        key = (key << 3 * bits) | (((x >> shift) & m) << 2 * bits) | (((y >> shift) & m) << bits) | ((z >> shift) & m)
    return key


def exact(case, seed):
    kind = case["kind"]
    if kind == "fit" and not case["bf16"]:
        # the loss also has the voxels that no Gaussian's kernel reaches: it is left out
        _, _, grads = _fit_grads(_inputs(case, seed), _inputs(case, int(seed) + 500_009), case["raw"], case["vs"], COLOR_WEIGHT)
        return {"loss": None, "density": None, "color": None, "grads": grads}
    if kind == "batch_fit" and case["n"] <= 600_000:
        t, other = _inputs(case, seed), _inputs(case, int(seed) + 500_009)
        start, _, vs = _batch_layout(case)
        total, parts = 0.0, []
        for a, b, v in zip(start[:-1], start[1:], vs):
            loss, missing, grads = _fit_grads(*[{k: x[k][int(a): int(b)] for k in NAMES} for x in (t, other)], case["raw"], float(v), 0.0)
            total += float(loss + missing)
            parts.append(grads)
        return {"loss": total, "density": None, "grads": {k: torch.cat([p[k] for p in parts]) for k in NAMES}}
    # topology is decided in 32 bits: in a large cloud a voxel on an ellipsoid's edge falls differently in 64
    if kind == "forward" and not case["window"] and not case["bf16"] and case["n"] <= 20_000:
        density = _forward_density(_inputs(case, seed), case["raw"], case["vs"])
        full = torch.zeros(_capacity(case)[1], dtype=torch.float64, device="cuda")
        full[: density.numel()] = density
        return {"grid": None, "density": full}
    return None
