"""The waits inside a map build's scans: when an earlier tile's sum does not arrive, every warp that
waits for it gives up together, the call reports it, and the context builds the next map as if
nothing had been."""
import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi

pytestmark = pytest.mark.gpu


def cloud(n, seed=1):
    # about one point in two cells: every scan of the build has several tiles
    rng = np.random.default_rng(seed)
    p = rng.uniform(0.0, 1.0, (n, 3)) * [400.0, 400.0, 20.0]
    return p.astype(np.float32)


def describe(ctx):
    i = ctx.map_info()
    return [i.num_points, i.num_segments, i.num_voxels, i.hash_capacity]


def test_segment_starts_give_up(gpu):
    p = cloud(200_000)
    ctx = capi.Context(resolution=2.0, min_points_per_voxel=2)
    ctx.set_target(p)
    want = describe(ctx)
    ctx.debug_lookback_stall(1_000_000, 2)  # 1 ms
    with pytest.raises(capi.NdtError, match="look-back"):
        ctx.set_target(p)
    ctx.debug_lookback_stall(0, 0)
    ctx.set_target(p)
    assert describe(ctx) == want


@pytest.mark.parametrize("kind", [1, 2, 3, 4])
def test_target_build_reports(gpu, kind):
    p = cloud(200_000, 2)
    ctx = capi.Context(resolution=2.0, min_points_per_voxel=2)
    ctx.set_target(p)
    want = describe(ctx)
    ctx.debug_lookback_stall(1_000_000, kind)
    with pytest.raises(capi.NdtError, match="look-back"):
        ctx.set_target(p)
    ctx.debug_lookback_stall(0, 0)
    ctx.set_target(p)
    assert describe(ctx) == want


@pytest.mark.parametrize("kind", [1, 2, 3])
def test_tile_put_reports(gpu, kind):
    p = cloud(200_000, 3)
    ctx = capi.Context(resolution=2.0, min_points_per_voxel=2)
    ctx.tile_put(1, p)
    ctx.tiles_commit()
    want = describe(ctx)
    ctx.debug_lookback_stall(1_000_000, kind)
    with pytest.raises(capi.NdtError, match="look-back"):
        ctx.tile_put(1, p)
    ctx.debug_lookback_stall(0, 0)
    ctx.tile_put(1, p)
    ctx.tiles_commit()
    assert describe(ctx) == want


@pytest.mark.parametrize("kind", [1, 2, 4])
def test_merge_reports(gpu, kind):
    p = cloud(200_000, 4)
    ctx = capi.Context(resolution=2.0, min_points_per_voxel=2)
    # whole cells a tile: y = 200 is a cell's edge
    ctx.tile_put(1, np.ascontiguousarray(p[p[:, 1] < 200]))
    ctx.tile_put(2, np.ascontiguousarray(p[p[:, 1] >= 200]))
    ctx.tiles_commit()
    want = describe(ctx)
    ctx.debug_lookback_stall(1_000_000, kind)
    with pytest.raises(capi.NdtError, match="look-back"):
        ctx.tiles_commit()
    assert describe(ctx) == want  # the map in use is still the old one
    ctx.debug_lookback_stall(0, 0)
    ctx.tiles_commit()
    assert describe(ctx) == want
