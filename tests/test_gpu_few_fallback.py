"""A few scans where the kernel that needs all its CTAs resident together is refused at its launch (the
rules go by more SMs than the device has, as on a context limited to part of them): the call takes the
cluster kernel of the same partition, and so do later calls, captured and asynchronous ones too."""
import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [0, 1])
def test_clusters_serve(gpu, graph):
    w = synth.queue_scans(seed=57, n_scans=8, lo=20_000, hi=24_000)
    poses = w.true_poses.copy()
    poses[:, 0] += 0.1
    res = []
    for form in (0, -1):
        ctx = capi.Context(max_iterations=5, work_queue=form, cuda_graph=graph)
        ctx.set_target(w.map_points)
        ctx.debug_sm_count(600)
        calls = [ctx.align_batch(w.scans, poses) for _ in range(3)]
        calls.append(ctx.batch_wait(ctx.batch_submit(w.scans, poses)))
        calls.append([ctx.align(w.scans[0], poses[0])])
        res.append(calls)
        ctx.debug_sm_count(0)
        ctx.align_batch(w.scans, poses)
    for a, b in zip(*res):
        for x, y in zip(a, b):
            for k in x:
                assert np.array_equal(x[k], y[k]), k
