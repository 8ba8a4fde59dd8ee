"""Voxels of one point (no covariance: no voxel, whatever min_points_per_voxel allows), of two equal
points (a zero covariance: no voxel either) and of two distinct ones, against the oracle: the same
voxels, counts and means bit for bit, covariances to f32 rounding."""
import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi

pytestmark = pytest.mark.gpu


def cloud(seed, offset):
    rng = np.random.default_rng(seed)
    one = rng.uniform(-300, 300, (2000, 3)) * [1, 1, 0.1]
    two = rng.uniform(-300, 300, (500, 3))
    same = rng.uniform(-300, 300, (300, 3))
    many = rng.normal(0, 0.3, (3000, 3)) + rng.uniform(-200, 200, (1, 3))
    p = np.concatenate([one, two, two + rng.normal(0, 0.02, two.shape), same, same, many])
    return (p + offset).astype(np.float32)


@pytest.mark.parametrize("min_points", [0, 1, 2, 3])
@pytest.mark.parametrize("offset", [0.0, -4001.25])
def test_against_oracle(gpu, oracle, min_points, offset):
    p = cloud(11, offset)
    ctx = capi.Context(resolution=2.0, min_points_per_voxel=min_points)
    ctx.set_target(p)
    g = oracle.Grid(p, 2.0, min_points=min_points)
    coords, means, covs, icovs, counts = ctx.map_voxels()
    assert np.array_equal(coords, g.coords)
    assert np.array_equal(counts, g.counts)
    assert np.array_equal(means, g.means)
    scale = np.abs(g.covs).max(1, keepdims=True)
    # FP64 sums and eigen-decomposition on both sides, rounded to f32 once
    assert (np.abs(covs.reshape(-1, 9) - g.covs) <= 2.0**-22 * scale).all()
    assert np.isfinite(icovs).all()
