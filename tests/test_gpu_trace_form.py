"""A traced call runs the kernel that the same call runs untraced: its results are the untraced ones bit
for bit, and its records are those of the cluster kernel up to the order of FP64 sums."""
import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("semantics", [0, 1])
@pytest.mark.parametrize("scans,points", [(1, 5000), (6, 700), (100, 1500)])
def test_traced_as_untraced(gpu, semantics, scans, points):
    w = synth.queue_scans(seed=53, n_scans=4, lo=5000, hi=6000)
    cut = [np.ascontiguousarray(w.scans[i % 4][:points + i]) for i in range(scans)]
    poses = w.true_poses[np.arange(scans) % 4].copy()
    poses[:, 0] += 0.1
    rec, res = [], []
    for form, trace in ((0, False), (0, True), (-1, True)):
        ctx = capi.Context(semantics=semantics, max_iterations=4, work_queue=form)
        ctx.set_target(w.map_points)
        ctx.trace(trace)
        res.append(ctx.align_batch(cut, poses))
        rec.append([ctx.read_trace(i) for i in range(scans)] if trace else None)
    for a, b in zip(res[0], res[1]):
        for k in a:
            assert np.array_equal(a[k], b[k]), k
    for i in range(scans):
        t, c = rec[1][i], rec[2][i]
        assert len(t) == res[0][i]["iterations"]
        # the first iteration: same pose, same lanes' f32 sums, FP64 sums in another order
        assert t[0, 0] == c[0, 0] and t[0, 2] == c[0, 2]
        assert np.array_equal(t[0, 3:9], c[0, 3:9])
        assert abs(t[0, 1] - c[0, 1]) <= 1e-13 * abs(c[0, 1])
        for lo, hi in ((9, 15), (15, 36)):
            scale = np.abs(c[0, 15:36]).max()
            assert np.abs(t[0, lo:hi] - c[0, lo:hi]).max() <= 1e-11 * scale
