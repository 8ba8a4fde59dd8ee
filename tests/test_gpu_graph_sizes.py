"""Captured batches of equally many scans with the same largest one but otherwise other sizes: a graph
captured for one large scan among small ones (a small grid, few points in all) must not serve a batch
of large scans. Times are held against an uncaptured context's on the same batch."""
import ctypes as C

import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi, synth

pytestmark = pytest.mark.gpu


def test_grid_of_the_batch_at_hand(gpu):
    import torch
    w = synth.queue_scans(seed=71, n_scans=8, lo=8000, hi=9000)
    n = min(len(s) for s in w.scans)
    large = [w.scans[i % 8][:n] for i in range(60)]
    small = [w.scans[0][:n]] + [w.scans[i % 8][:30] for i in range(59)]
    poses = w.true_poses[np.arange(60) % 8].copy()
    poses[:, 0] += 0.1
    res = (capi.Result * 60)()
    dev = []
    for cut in (small, large):
        xyz = torch.from_numpy(np.concatenate(cut).astype(np.float32)).cuda()
        dev.append((xyz, np.concatenate([[0], np.cumsum([len(s) for s in cut])]).astype(np.uint64)))
    ms, out = [], []
    for graph in (0, 1):
        ctx = capi.Context(max_iterations=5, work_queue=4, cuda_graph=graph)
        ctx.set_target(w.map_points)

        def run(k):
            xyz, off = dev[k]
            capi.check(ctx.lib.ndt_align_batch_device(ctx.h, C.c_void_p(xyz.data_ptr()),
                                                      off.ctypes.data, poses.ctypes.data, 60, res))
        run(0)
        t = []
        for _ in range(15):
            before = ctx.stats()["align_kernel_ms"]
            run(1)
            t.append(ctx.stats()["align_kernel_ms"] - before)
        ms.append(np.median(t))
        out.append(bytes(res))
    assert out[0] == out[1]
    # 16 chunks against 300: the small grid takes several times as long
    assert ms[1] <= 1.3 * ms[0], ms


def test_withheld_launch_is_not_captured(gpu):
    w = synth.queue_scans(seed=73, n_scans=4, lo=2000, hi=3000)
    ctx = capi.Context(max_iterations=3, work_queue=2, cuda_graph=1)
    ctx.set_target(w.map_points)
    ctx.debug_queue_stall(1_000_000, withhold_next=True)
    with pytest.raises(capi.NdtError):
        ctx.align_batch(w.scans, w.true_poses)
    a = ctx.align_batch(w.scans, w.true_poses)
    ctx.debug_queue_stall(0)
    b = ctx.align_batch(w.scans, w.true_poses)
    for x, y in zip(a, b):
        assert np.array_equal(x["pose"], y["pose"])
