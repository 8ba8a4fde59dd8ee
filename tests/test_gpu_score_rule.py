"""The scoring kernel at every number of points per thread that its rule gives (1, 2, 4, 8 by the points
in all; more where scans of uneven size would leave the grid empty), with the dense index and with
the hash: FP64 sums of the same f32 terms whatever the split."""
import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi

pytestmark = pytest.mark.gpu

# positive terms, so a sum's error is relative: a term passes at most 28 additions (8 a thread, 5
# and 8 in the block, 2 and 5 over the blocks), each rounded to 2^-53, on either side
TOL = 2 * 28 * 2.0**-53


@pytest.mark.parametrize("cell_index", [0, 1])
def test_sums_do_not_depend_on_the_split(gpu, single_cases, oracle, cell_index):
    case = single_cases[1]
    ctx = capi.Context(cell_index=cell_index)
    ctx.set_target(case.map_points)
    rng = np.random.default_rng(4)
    scan = np.ascontiguousarray(case.scan[rng.integers(0, len(case.scan), 9000)])
    T = oracle.pose_T34_zyx(case.true_pose)
    want = None
    # 9,000 points at 1 pose up to 4.5M in all
    for poses in (1, 16, 17, 50, 51, 200, 438, 439, 500):
        Ts = np.tile(np.asarray(T).reshape(1, -1), (poses, 1))
        nvtl, tp = ctx.eval_batch(scan, Ts)
        assert (nvtl == nvtl[0]).all() and (tp == tp[0]).all()
        if want is None:
            want = nvtl[0], tp[0]
            ref = oracle.Grid(case.map_points, 2.0).nvtl(scan, T)
            assert abs(nvtl[0] - ref) <= 1e-5 * abs(ref)
        assert abs(nvtl[0] - want[0]) <= TOL * want[0]
        assert abs(tp[0] - want[1]) <= TOL * want[1]


def test_uneven_scans(gpu, single_cases):
    """One large scan among many small ones: each scan's NVTL is the one it gets alone."""
    case = single_cases[0]
    ctx = capi.Context(max_iterations=1)
    ctx.set_target(case.map_points)
    rng = np.random.default_rng(6)
    scans = [np.ascontiguousarray(case.scan[rng.integers(0, len(case.scan), n)])
             for n in [60_000] + [40 + i for i in range(300)]]
    got = ctx.align_batch(scans, [case.guess] * len(scans))
    for i in (0, 1, 150, 300):
        one = ctx.align_batch([scans[i]], [case.guess])[0]
        # the poses differ by the order of FP64 sums (at most 1e-9 after one iteration)
        assert abs(one["nvtl"] - got[i]["nvtl"]) <= 1e-7 * abs(one["nvtl"])
