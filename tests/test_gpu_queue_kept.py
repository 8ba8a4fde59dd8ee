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
    cluster = capi.Context(max_iterations=3, work_queue=-1)
    cluster.set_target(w.map_points)
    shared = capi.Context(max_iterations=3)
    shared.set_target(w.map_points)
    res = (capi.Result * scans)()
    want = []
    for arr, _, _ in batches:
        cluster.align_batch_raw(arr, res)
        counts = [(r.iterations, r.status, r.num_correspondences) for r in res]
        alone = capi.Context(max_iterations=3)  # a context that has seen no other batch
        alone.set_target(w.map_points)
        C.memset(res, 0xFF, C.sizeof(res))
        alone.align_batch_raw(arr, res)
        assert [(r.iterations, r.status, r.num_correspondences) for r in res] == counts
        want.append(bytes(res))
    for turn in range(40):
        C.memset(res, 0xFF, C.sizeof(res))
        shared.align_batch_raw(batches[turn % 2][0], res)
        assert bytes(res) == want[turn % 2], turn


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("queue,iterations,scans", [(1, 5, 330), (2, 5, 500), (4, 10, 310),
                                                    (2, 30, 1300)])
def test_kept_alignments_of_several_chunks(gpu, queue, iterations, scans, graph):
    """Who sums a chunk does not matter: a batch large enough for its CTAs to keep their alignments
    gives each scan the result that it gets in a small batch, whose chunks any CTA claims."""
    w = synth.queue_scans(seed=61, n_scans=8, lo=4000, hi=5000)
    size = [1 + (371 * i) % 2048 for i in range(scans)]
    size[0] = 2048
    cut = [np.ascontiguousarray(w.scans[i % 8][i % 40:i % 40 + n]) for i, n in enumerate(size)]
    poses = w.true_poses[np.arange(scans) % 8].copy()
    poses[:, 0] += 0.1
    ctx = capi.Context(max_iterations=iterations, work_queue=queue, cuda_graph=graph)
    ctx.set_target(w.map_points)
    both = []
    for parts in ([slice(0, scans)], [slice(i, i + 100) for i in range(0, scans, 100)]):
        got = []
        for s in parts:
            got += ctx.align_batch(cut[s], poses[s])
        both.append(got)
    for i, (a, b) in enumerate(zip(*both)):
        for k in ("pose", "score", "hessian", "iterations", "status", "num_correspondences"):
            assert np.array_equal(a[k], b[k]), (i, size[i], k)
