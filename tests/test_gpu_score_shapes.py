"""The scoring kernel at the edges of its blocks and of its points-per-thread rule: point counts
around one block of 128 threads, one to many poses (the grid decides how many points a thread
takes and whether a job's blocks are summed by its last block)."""
import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi

pytestmark = pytest.mark.gpu

# f32 terms (relative error about 1e-6 each, d2 sq / 2 below 10) against FP64
REL = 1e-5


@pytest.fixture(scope="module")
def setup(oracle, single_cases):
    case = single_cases[0]
    ctx = capi.Context()
    ctx.set_target(case.map_points)
    rng = np.random.default_rng(4)
    scan = case.scan[rng.integers(0, len(case.scan), 9000)]
    Ts = []
    for _ in range(600):
        p = case.true_pose.copy()
        p[:2] += rng.uniform(-0.3, 0.3, 2)
        p[5] += rng.uniform(-0.02, 0.02)
        Ts.append(oracle.pose_T34_zyx(p))
    return ctx, oracle.Grid(case.map_points, 2.0), scan, np.array(Ts)


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 256, 257, 1025, 9000])
@pytest.mark.parametrize("poses", [1, 3, 600])
def test_nvtl_at_block_edges(gpu, setup, n, poses):
    ctx, grid, scan, Ts = setup
    nvtl, tp = ctx.eval_batch(scan[:n], Ts[:poses])
    for k in sorted({0, poses // 2, poses - 1}):
        want = grid.nvtl(scan[:n], Ts[k])
        assert abs(nvtl[k] - want) <= REL * abs(want)
    # the same call again: the finished-block counters were left at zero
    again, tp2 = ctx.eval_batch(scan[:n], Ts[:poses])
    assert np.array_equal(nvtl, again) and np.array_equal(tp, tp2)


def test_single_pose_equals_many(gpu, setup):
    """A pose scored alone (one point per thread) and among many (several): sums of the same
    f32 terms, so they agree to the 48 bits they are carried in."""
    ctx, _, scan, Ts = setup
    many, tp_many = ctx.eval_batch(scan, Ts)
    one, tp_one = ctx.eval_batch(scan, Ts[:1])
    assert abs(many[0] - one[0]) <= 1e-12 * abs(one[0])
    assert abs(tp_many[0] - tp_one[0]) <= 1e-12 * abs(tp_one[0])


def test_empty_scan(gpu, setup):
    ctx, _, scan, Ts = setup
    nvtl, tp = ctx.eval_batch(scan[:0], Ts[:3])
    assert not nvtl.any() and not tp.any()
