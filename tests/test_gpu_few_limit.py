"""The waits between the CTAs of the few-alignments kernel: with a limit that no exchange can meet the
call reports it, and the context aligns as before once the limit is restored."""
import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi, synth

pytestmark = pytest.mark.gpu


def test_wait_runs_out(gpu):
    w = synth.queue_scans(seed=79, n_scans=4, lo=5000, hi=6000)
    poses = w.true_poses.copy()
    poses[:, 0] += 0.1
    ctx = capi.Context(max_iterations=6)
    ctx.set_target(w.map_points)
    want = ctx.align_batch(w.scans, poses)
    ctx.debug_queue_stall(1)  # 1 ns: a frame is never there that soon
    with pytest.raises(capi.NdtError):
        for _ in range(3):
            ctx.align_batch(w.scans, poses)
    ctx.debug_queue_stall(0)
    for _ in range(2):
        for a, b in zip(ctx.align_batch(w.scans, poses), want):
            for k in a:
                assert np.array_equal(a[k], b[k]), k
