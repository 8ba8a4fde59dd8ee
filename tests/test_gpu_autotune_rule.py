"""The autotuner times the form that an untuned call takes beside the others: tuning a class of a few
scans must not put its calls on a slower form. A tuned call's kernel time is held against an untuned
one's on the same batch, medians of many calls in turn; the candidates differ by factors (a 20k-point
scan 127 us on all SMs, 297 on a cluster), run-to-run noise is below 2%."""
import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scans,points", [(1, 6000), (8, 4000), (30, 1500), (400, 1500)])
def test_tuned_is_not_slower(gpu, scans, points):
    import torch
    w = synth.queue_scans(seed=51, n_scans=8, lo=6000, hi=8000)
    cut = [w.scans[i % 8][:points] for i in range(scans)]
    xyz = torch.from_numpy(np.concatenate(cut).astype(np.float32)).cuda()
    offsets = np.concatenate([[0], np.cumsum([len(s) for s in cut])]).astype(np.uint64)
    poses = w.true_poses[np.arange(scans) % 8].copy()
    poses[:, 0] += 0.1
    ctxs = [capi.Context(max_iterations=8) for _ in range(2)]
    for c in ctxs:
        c.set_target(w.map_points)
    r = ctxs[1].autotune(xyz.data_ptr(), offsets, poses, repeats=3)
    assert r["candidates"] == 46
    ms = [[], []]
    for _ in range(25):
        for k, c in enumerate(ctxs):
            before = c.stats()["align_kernel_ms"]
            c.align_batch_device(xyz.data_ptr(), offsets, list(poses))
            ms[k].append(c.stats()["align_kernel_ms"] - before)
    untuned, tuned = (float(np.median(m[5:])) for m in ms)
    print(f"{scans} x {points}: untuned {untuned:.4f} ms, tuned {tuned:.4f} ms ({r})")
    assert tuned <= 1.1 * untuned
