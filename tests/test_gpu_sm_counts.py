"""The rules that go by the SM count (points per thread of the scoring kernel, CTAs that stay to the end
of a batch, launch shapes) at counts below and at the device's: alignments and scores are those of
the device's own count up to the order of sums."""
import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sms", [1, 20, 76, 148])
def test_other_counts(gpu, sms):
    w = synth.queue_scans(seed=59, n_scans=8, lo=6000, hi=9000)
    poses = w.true_poses[np.arange(40) % 8].copy()
    poses[:, 0] += 0.05
    scans = [w.scans[i % 8] for i in range(40)]
    T = np.tile(np.eye(4)[:3].ravel(), (30, 1))
    T[:, 3] = np.linspace(-3, 3, 30)
    out = []
    for n in (0, sms):
        ctx = capi.Context(max_iterations=2, work_queue=2)
        ctx.set_target(w.map_points)
        ctx.debug_sm_count(n)
        r = ctx.align_batch(scans, poses)
        nvtl, tp = ctx.eval_batch(w.scans[0], T)
        out.append((r, nvtl, tp))
    for a, b in zip(out[0][0], out[1][0]):
        # one kernel and partition: the same bit for bit but for the scores' sums
        for k in ("pose", "score", "hessian", "iterations", "status", "num_correspondences"):
            assert np.array_equal(a[k], b[k]), k
        assert abs(a["nvtl"] - b["nvtl"]) <= 1e-12 * abs(b["nvtl"])
    assert np.abs(out[0][1] - out[1][1]).max() <= 1e-12
    assert np.abs(out[0][2] - out[1][2]).max() <= 1e-12
