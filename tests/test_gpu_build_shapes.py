"""The map build over box shapes and point counts at its edges: key widths of every kind (the sort
keys interleave only the bits that a box has), tiles of 4,096 keys and their remainders, non-finite
points, unaligned device input, against the oracle (voxel order, coordinates, counts and means bit
for bit)."""
import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi

pytestmark = pytest.mark.gpu

BOXES = {
    "line_x": (6000, 3, 3), "line_y": (3, 6000, 3), "line_z": (3, 3, 900),
    "plane_xy": (400, 300, 1), "plane_xz": (500, 1, 200), "plane_yz": (1, 300, 260),
    "cube": (60, 60, 60), "x_long": (1500, 90, 20), "y_long": (70, 1100, 30),
    "z_long": (30, 50, 700), "cell": (1, 1, 1), "two_cells": (3, 1, 1),
}


def cloud(extent, n, seed, offset=(0.0, 0.0, 0.0)):
    rng = np.random.default_rng(seed)
    ext = np.asarray(extent, float)
    centres = rng.uniform(0, 1, (max(1, n // 12), 3)) * ext
    p = centres[rng.integers(0, len(centres), n)] + rng.normal(0, 0.25, (n, 3))
    return (p + np.asarray(offset)).astype(np.float32)


def check(oracle, pts, res=2.0, device=None, cell_index=0):
    ctx = capi.Context(resolution=res, cell_index=cell_index)
    if oracle.Grid(pts, res).n == 0:  # too few points in any one cell
        with pytest.raises(capi.NdtError, match="No voxels"):
            ctx.set_target(pts)
        return None
    if device is None:
        ctx.set_target(pts)
    else:
        ctx.set_target_device(device, len(pts))
    g = oracle.Grid(pts, res)
    coords, means, covs, icovs, counts = ctx.map_voxels()
    assert np.array_equal(coords, g.coords)
    assert np.array_equal(counts, g.counts)
    assert np.array_equal(means, g.means)
    return ctx, g


@pytest.mark.parametrize("box", list(BOXES))
@pytest.mark.parametrize("offset", [(0, 0, 0), (-3001.5, 777.25, -40.0)])
def test_box_shapes(gpu, oracle, box, offset):
    check(oracle, cloud(BOXES[box], 30_011, 7, offset))


@pytest.mark.parametrize("n", [6, 7, 63, 4095, 4096, 4097, 8192, 65_537, 700_001])
def test_tile_edges(gpu, oracle, n):
    check(oracle, cloud((80, 80, 6), n, n))


@pytest.mark.parametrize("n", [5000, 4096 * 3 + 1])
def test_non_finite_points(gpu, oracle, n):
    pts = cloud((80, 80, 6), n, 3)
    pts[::7, 0] = np.nan
    pts[5::11, 2] = np.inf
    pts[-1] = -np.inf
    check(oracle, pts)


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_unaligned_device_points(gpu, oracle, shift):
    import torch
    pts = cloud((80, 80, 6), 20_003, 5)
    buf = torch.zeros(len(pts) * 3 + 8, device="cuda")
    buf[shift:shift + pts.size] = torch.tensor(pts.ravel(), device="cuda")
    torch.cuda.synchronize()
    check(oracle, pts, device=buf.data_ptr() + 4 * shift)


@pytest.mark.parametrize("cell_index", [0, 1, 2])
def test_search_forms_agree(gpu, oracle, cell_index):
    """Dense index (octant masks gathered per cell), hash, and NDT_CELL_INDEX_OCTANT list the
    oracle's neighbours."""
    pts = cloud((150, 120, 14), 60_000, 9)
    ctx, g = check(oracle, pts, cell_index=cell_index)
    rng = np.random.default_rng(1)
    q = (pts[rng.integers(0, len(pts), 4000)] + rng.normal(0, 1.5, (4000, 3))).astype(np.float32)
    idx, cnt = ctx.neighbors(q, 27)
    widx, wcnt = g.query_gpu_sem(q, 27)
    assert np.array_equal(cnt, wcnt) and np.array_equal(idx, widx)
