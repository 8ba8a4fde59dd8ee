"""The work-queue kernel under the most frequent change of chunks: thousands of scans of a few points,
so that a warp's unit, its chunk and the slot that holds it change every few hundred cycles. One
iteration's score, correspondence count and Hessian of every scan are the sums over its own points,
whichever warp summed them: compared with the cluster kernel's, and run to run."""
import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads,top", [(128, 40), (256, 700)])
def test_units_sum_their_own_points(gpu, threads, top):
    w = synth.queue_scans(seed=47, n_scans=8, lo=3000, hi=4000)
    m = 3000
    size = [1 + (7 * i) % top for i in range(m)]
    scans = [np.ascontiguousarray(w.scans[i % 8][i % 50:][:n]) for i, n in enumerate(size)]
    arr, _, _ = capi.scan_array(scans, w.true_poses[np.arange(m) % 8])
    out = []
    for form, t in ((-1, 0), (1, threads)):
        ctx = capi.Context(max_iterations=1, work_queue=form, threads_per_cta=t)
        ctx.set_target(w.map_points)
        res = (capi.Result * m)()
        ctx.align_batch_raw(arr, res)
        first = bytes(res)
        for _ in range(10):
            ctx.align_batch_raw(arr, res)
            assert bytes(res) == first
        out.append([(r.num_correspondences, r.score, np.array(r.hessian[:])) for r in res])
    for i, (a, b) in enumerate(zip(*out)):
        assert a[0] == b[0], i
        # a lane's f32 sums differ between the partitions: at most 8 points of 5 pairs a lane, each
        # rounded to 2^-24 of the largest term of the entry
        assert abs(a[1] - b[1]) <= 1e-5 * abs(a[1]), i
        assert np.abs(a[2] - b[2]).max() <= 1e-4 * np.abs(a[2]).max(), i
