"""The drop-in entries' walk, which evaluates the RGBA8 values alone, against the walk
that also sums the float channels: the same node2 bytes, values and header, on clouds
that reach its edges (opaque, stacked, one-voxel and far Gaussians, colours out of
range, an empty cloud), with and without the per-byte check on the device."""

import numpy as np
import pytest

from test_gpu_walk_sums import _cloud

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("check", [False, True])
@pytest.mark.parametrize("kind", ["colors", "opaque", "stack", "thin", "far", "culled"])
def test_bytes_of_both_walks(monkeypatch, kind, check):
    from nanovdb_editor import Compute, Raster
    from nanovdb_editor.grid import NodeGrid
    from nanovdb_editor.vox import FLAG_RAW_INPUTS, FLAG_WINDOW_ORDER, VoxContext

    if check:
        monkeypatch.setenv("VOX_CHECK_EMIT", "1")
    ctx = VoxContext(0)
    compute = Compute(device_index=0)
    raster = Raster(compute)
    for n, vs in ((1, 0.01), (13, 0.01), (700, 0.004), (3000, 0.01)):
        c = _cloud(kind, n, vs, n + 2)
        if kind == "culled":
            c["opacities"][:] = 0.005  # below the 0.01 cutoff: no pair at all
        means, logit, quats, log_s, sh0, _ = c.raw_arrays()
        want = ctx.voxelize_host(means, quats, log_s, logit, sh0, vs, 0.05, FLAG_RAW_INPUTS | FLAG_WINDOW_ORDER)
        arrays = [compute.create_array(np.ascontiguousarray(a)) for a in (means, logit, quats, log_s, sh0)]
        arrays.append(compute.create_array(np.zeros(0, np.float32)))
        result = raster.raster_to_nanovdb_from_arrays(vs, arrays)
        got = NodeGrid(np.array(compute.map_array(result, np.uint8)))
        for name in want.header.dtype.names:
            if name not in ("grid_bytes", "density_offset", "color_offset"):
                assert np.array_equal(got.header[name], want.header[name]), name
        assert np.array_equal(got.node2, want.node2) and np.array_equal(got.rgba8, want.rgba8)
        assert np.array_equal(got.bbox, want.bbox) and got.density is None and got.color is None
        for a in arrays + [result]:
            compute.destroy_array(a)
    ctx.close()
