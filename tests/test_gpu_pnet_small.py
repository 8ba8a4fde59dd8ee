"""Proposals for a few scans: short scans filled in by the calling thread, by the host threads and copied
as they lie, around the sizes where the rule changes (65,536 points), each scan's proposals those it
gets alone; one sample and as many as the GPU has SMs."""
import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [
    [65_535], [65_536], [65_537], [1, 65_536, 2], [65_535, 65_535], [40_000] * 9,
    [70_000, 10, 349_526, 65_535, 30, 66_000], [100] * 151, [100] * 153,
], ids=lambda s: f"{len(s)}x{s[0]}")
def test_alone_and_together(gpu, sizes):
    c = synth.single_case(2)
    net = capi.PNet(seed=9)
    mid = net.add_map(c.map_points)
    rng = np.random.default_rng(4)
    p = np.concatenate([c.scan] * (1 + max(sizes) // len(c.scan)))
    scans = [np.ascontiguousarray(p[rng.permutation(len(p))[:n]]) for n in sizes]
    coarse = np.tile(np.asarray(c.guess, float), (len(scans), 1))
    coarse[:, 5] += np.arange(len(scans)) * 0.01
    poses, logits = net.propose(mid, scans, coarse)
    for i in {0, len(scans) // 2, len(scans) - 1}:
        one = net.propose(mid, [scans[i]], coarse[i:i + 1])
        assert np.array_equal(one[0][0], poses[i]) and np.array_equal(one[1][0], logits[i])
