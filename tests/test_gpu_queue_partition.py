"""Batches on the work-queue kernel with a cluster's partition of the points (the default for
more than a few scans) against the same batch on the cluster kernel: every lane sums the same
points in the same order, so only the order of FP64 sums differs. Sizes sit at the partition's
edges (warps without points, one point more than a warp, a CTA, a cluster) and include empty and
partly non-finite scans; a batch of small scans takes the form in which a CTA keeps its
alignments, a large batch of large scans is copied in while the kernel runs."""
import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi, synth

pytestmark = pytest.mark.gpu

# three iterations from 0.1 m: an FP64 rounding (1e-16 of a step) grows by far less than 1e5
TOL = 1e-10


@pytest.fixture(scope="module")
def workload():
    w = synth.queue_scans(seed=41, n_scans=12, lo=30_000, hi=40_000)
    rng = np.random.default_rng(3)
    poses = w.true_poses.copy()
    poses[:, :2] += rng.uniform(-0.1, 0.1, (12, 2))
    return w, poses


def both(workload, sizes, semantics, graph=0, order=None):
    w, poses = workload
    scans, guess = [], []
    for i, n in enumerate(sizes):
        s = w.scans[i % 12]
        scans.append(np.ascontiguousarray(s[:n] if n <= len(s) else s))
        guess.append(poses[i % 12])
    if len(scans) > 3 and len(scans[2]) > 40:
        scans[2] = scans[2].copy()
        scans[2][7] = np.nan
        scans[2][33, 1] = np.inf
    out = []
    for form in (0, -1):
        ctx = capi.Context(semantics=semantics, max_iterations=3, work_queue=form,
                           cuda_graph=graph)
        ctx.set_target(w.map_points)
        a = ctx.align_batch(scans, guess)
        b = ctx.align_batch(scans, guess)
        for x, y in zip(a, b):
            assert np.array_equal(x["pose"], y["pose"]) and x["score"] == y["score"]
        out.append(a)
    for i, (x, y) in enumerate(zip(*out)):
        for k in ("iterations", "num_correspondences", "status", "converged"):
            assert x[k] == y[k], (i, sizes[i], k)
        assert np.abs(x["pose"] - y["pose"]).max() <= TOL, (i, sizes[i])
        scale = np.abs(y["hessian"]).max() + 1e-300
        assert np.abs(x["hessian"] - y["hessian"]).max() <= TOL * scale, (i, sizes[i])
        assert abs(x["score"] - y["score"]) <= TOL * abs(y["score"])


@pytest.mark.parametrize("semantics", [0, 1])
@pytest.mark.parametrize("sizes", [
    [0, 1, 31, 32, 33, 100, 127, 128, 129, 255],
    [1023, 1024, 1025, 511, 512, 513, 2049, 700, 900, 20],
    [4095, 4096, 4097, 8191, 30_000, 5000, 12_289, 40_000, 1, 0, 6000, 64],
], ids=["T128", "T256", "T512"])
def test_default_batch_equals_cluster_kernel(gpu, workload, sizes, semantics):
    both(workload, sizes, semantics)


@pytest.mark.parametrize("graph", [0, 1])
def test_ctas_keep_their_alignments(gpu, workload, graph):
    """More single-chunk alignments than the grid has CTAs."""
    both(workload, [1024 + 13 * (i % 70) for i in range(1500)], 0, graph)


def test_large_batch_streams_in(gpu, workload):
    both(workload, [20_000 + 37 * i for i in range(70)], 0)
