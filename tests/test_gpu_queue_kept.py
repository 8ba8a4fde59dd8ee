"""Batches in which a CTA of the work-queue kernel keeps its alignments from the first iteration to
the last: no alignment may be left behind by a CTA that leaves early. Two different batches take
turns on one context, so a result that a call did not write would be the other batch's; sizes make
the kernel take and finish thousands of alignments a call, with CTAs leaving while others step."""
import ctypes as C

import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scans,points", [(1400, 1024), (3200, 1100), (700, 2040)])
def test_no_alignment_is_left_behind(gpu, scans, points):
    w = synth.queue_scans(seed=43, n_scans=8, lo=4000, hi=5000)
    rng = np.random.default_rng(5)
    batches = []
    for b in range(2):
        poses = w.true_poses[np.arange(scans) % 8].copy()
        poses[:, :2] += rng.uniform(-0.1, 0.1, (scans, 2))
        cut = [np.ascontiguousarray(w.scans[(i + b) % 8][b:b + points + i % 3])
               for i in range(scans)]
        poses = poses if b == 0 else poses[(np.arange(scans) + 1) % scans]
        batches.append(capi.scan_array(cut, poses))
    want = None
    for form in (-1, 0):
        ctx = capi.Context(max_iterations=3, work_queue=form)
        ctx.set_target(w.map_points)
        res = (capi.Result * scans)()
        if form == -1:
            want = []
            for arr, _, _ in batches:
                ctx.align_batch_raw(arr, res)
                want.append([(r.iterations, r.status, r.num_correspondences, r.pose[0])
                             for r in res])
            continue
        first = [None, None]
        for turn in range(40):
            b = turn % 2
            C.memset(res, 0xFF, C.sizeof(res))
            ctx.align_batch_raw(batches[b][0], res)
            got = bytes(res)
            if first[b] is None:
                first[b] = got
                # the cluster kernel's lanes sum the same points, FP64 sums in another order: three
                # iterations from 0.1 m grow a rounding of 1e-16 by far less than 1e6
                for i, (r, x) in enumerate(zip(res, want[b])):
                    assert (r.iterations, r.status, r.num_correspondences) == x[:3], (b, i)
                    assert abs(r.pose[0] - x[3]) <= 1e-10, (b, i)
            assert got == first[b], (turn, b)
