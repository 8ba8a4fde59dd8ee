"""Host arrays that reach the proposal network through pinned halves of 4 MB: results do not
depend on how the scans fall into halves, batches and pieces, and parameters come out as they
went in."""
import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def net():
    c = synth.single_case(1)
    n = capi.PNet(seed=5)
    return n, n.add_map(c.map_points), c


def scans_of(c, sizes):
    rng = np.random.default_rng(1)
    p = np.concatenate([c.scan] * (1 + max(sizes) // len(c.scan)))
    return [np.ascontiguousarray(p[rng.permutation(len(p))[:n]]) for n in sizes]


@pytest.mark.parametrize("sizes", [
    [1], [349_525], [349_526], [1_200_000],                # a half holds 349,525.3 points
    [100, 700_000, 3, 349_000, 50],                        # ranges across halves
    [1 + 7 * (i % 50) for i in range(300)],                # more queries than a batch
], ids=["1", "half", "half+", "long", "ragged", "300"])
def test_propose_staging(gpu, net, sizes):
    n, mid, c = net
    scans = scans_of(c, sizes)
    coarse = np.tile(np.asarray(c.guess, float), (len(scans), 1))
    coarse[:, 5] += np.arange(len(scans)) * 0.01
    poses, logits = n.propose(mid, scans, coarse)
    # the order of a scan's points does not matter to its grid
    again = n.propose(mid, [np.ascontiguousarray(s[::-1]) for s in scans], coarse)
    assert np.array_equal(poses, again[0]) and np.array_equal(logits, again[1])
    for i in {0, len(scans) // 2, len(scans) - 1}:
        one = n.propose(mid, [scans[i]], coarse[i:i + 1])
        assert np.array_equal(one[0][0], poses[i]) and np.array_equal(one[1][0], logits[i])


def test_params_round_trip(gpu, net):
    n = net[0]
    v = np.random.default_rng(2).normal(size=len(n.params())).astype(np.float32)
    n.set_params(v)
    assert np.array_equal(n.params(), v)
