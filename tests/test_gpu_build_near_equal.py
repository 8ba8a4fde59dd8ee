"""Voxels whose two largest eigenvalues are equal or nearly so (1e-9 to 1e-5 apart): the clamp's
threshold is a hundredth of the largest in FP64, so covariances stay within 2 and inverses within 4
f32 ULP of the oracle's FP64 build, the bounds of every other map."""
import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi
from parity_helpers import matrix_ulps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flat", [0.0, 1e-3, 0.03])
def test_flat_squares(gpu, oracle, flat):
    rng = np.random.default_rng(3)
    m = 1500
    u = np.linspace(-0.9, 0.9, 7)
    gx, gy = (a.ravel() for a in np.meshgrid(u, u))
    pts = []
    for i in range(m):
        d = 10.0 ** rng.uniform(-9, -5) if i % 3 else 0.0
        z = flat * rng.normal(0, 1, gx.size)
        q, _ = np.linalg.qr(rng.normal(0, 1, (3, 3)))
        p = np.stack([gx * 0.5, gy * 0.5 * (1 + d), z], 1) @ q.T
        pts.append(p + 2.0 * np.array([i % 50, i // 50, 0]) + 1.0)
    p = np.concatenate(pts).astype(np.float32)
    ctx = capi.Context(resolution=2.0)
    ctx.set_target(p)
    g = oracle.Grid(p, 2.0)
    coords, means, covs, icovs, counts = ctx.map_voxels()
    assert np.array_equal(coords, g.coords) and np.array_equal(counts, g.counts)
    assert np.array_equal(means, g.means)
    assert matrix_ulps(covs, g.covs).max() <= 2.0
    assert matrix_ulps(icovs, g.icovs).max() <= 4.0
