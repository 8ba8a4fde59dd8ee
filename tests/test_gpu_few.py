"""Few alignments spread over the GPU (the default for up to eight scans or a small batch)
against the same call on the cluster kernel: every lane sums the same points in the same order,
so only the order of FP64 sums differs. Sizes sit at the edges of warps, item batches and CTA
shares and include empty and partly non-finite scans. Batches that reach the work-queue kernel
by the default rule, with several partition ranks, are compared the same way."""
import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi, synth

pytestmark = pytest.mark.gpu

# three iterations from 0.1 m: an FP64 rounding (1e-16 of a step) grows by far less than 1e5
TOL = 1e-10


@pytest.fixture(scope="module")
def workload():
    w = synth.queue_scans(seed=43, n_scans=4, lo=40_000, hi=40_000)
    rng = np.random.default_rng(5)
    poses = w.true_poses.copy()
    poses[:, :2] += rng.uniform(-0.1, 0.1, (4, 2))
    return w, poses


def both(workload, sizes, **options):
    w, poses = workload
    scans, guess = [], []
    for i, n in enumerate(sizes):
        s = np.concatenate([w.scans[i % 4]] * (1 + n // 40_000))[:n].copy()
        if n > 40:
            s[7] = np.nan
            s[33, 1] = np.inf
        scans.append(s)
        guess.append(poses[i % 4])
    out = []
    for form in (0, -1):
        ctx = capi.Context(max_iterations=3, work_queue=form, **options)
        ctx.set_target(w.map_points)
        a = ctx.align_batch(scans, guess)
        b = ctx.align_batch(scans, guess)
        for x, y in zip(a, b):
            assert np.array_equal(x["pose"], y["pose"]) and x["score"] == y["score"]
        out.append(a)
    for i, (x, y) in enumerate(zip(*out)):
        for k in ("iterations", "num_correspondences", "status", "converged",
                  "oscillation_count"):
            assert x[k] == y[k], (i, sizes[i], k)
        assert np.abs(x["pose"] - y["pose"]).max() <= TOL, (i, sizes[i])
        scale = np.abs(y["hessian"]).max() + 1e-300
        assert np.abs(x["hessian"] - y["hessian"]).max() <= TOL * scale, (i, sizes[i])
        assert abs(x["score"] - y["score"]) <= TOL * abs(y["score"])


@pytest.mark.parametrize("semantics", [0, 1])
@pytest.mark.parametrize("n", [0, 1, 31, 32, 33, 127, 129, 1023, 1024, 2047, 4095, 4097, 12_289,
                               40_000, 120_001])
def test_one_scan(gpu, workload, n, semantics):
    both(workload, [n], semantics=semantics)


@pytest.mark.parametrize("options", [{}, {"cuda_graph": 1}, {"max_neighbors": 27},
                                     {"semantics": 1}], ids=str)
@pytest.mark.parametrize("sizes", [
    [40_000, 0],
    [16_384, 520, 33, 5000, 1, 0, 100_000, 4096],
    [1500] * 48,
    # 113 scans of 17 warps with one or two CTAs each (more warps than a CTA takes at a time)
    [16_384] + [520] * 113,
], ids=["2", "8", "48", "114"])
def test_several_scans(gpu, workload, sizes, options):
    both(workload, sizes, **options)


@pytest.mark.parametrize("graph", [0, 1])
def test_large_batch_of_clusters(gpu, workload, graph):
    """More than 1.75 waves of clusters: the work-queue kernel, several ranks a scan."""
    edges = [4096, 4097, 8191, 1023, 512, 33, 1, 0, 12_289, 5000]
    both(workload, [edges[i % 10] if i < 40 else 4200 + 7 * i for i in range(120)],
         cuda_graph=graph)
