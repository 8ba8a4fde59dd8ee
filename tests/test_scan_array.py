"""The C array of scans and poses, filled by columns or element by element, is the same."""
import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi


def fields(arr):
    return [(s.num_points, list(s.initial_pose)) for s in arr]


@pytest.mark.parametrize("make", [
    lambda p: p, lambda p: [tuple(r) for r in p], lambda p: p.astype(np.float32),
    lambda p: np.asfortranarray(p), lambda p: np.hstack([p, p]), lambda p: np.vstack([p, p]),
    lambda p: p.astype(int), lambda p: [[str(x) for x in r] for r in p],
    lambda p: [list(p[0]) + [9.0]] + [list(r) for r in p[1:]], lambda p: p.astype(object)])
def test_poses(make):
    rng = np.random.default_rng(0)
    scans = [rng.random((3 + i, 3)).astype(np.float32) for i in range(4)]
    poses = make(rng.normal(size=(4, 6)) * 10)
    arr, m, keep = capi.scan_array(scans, poses)
    assert m == 4
    assert fields(arr) == [(3 + i, [float(poses[i][k]) for k in range(6)]) for i in range(4)]
    assert [s.xyz for s in arr] == [k.ctypes.data for k in keep]


def test_scans_that_need_a_copy():
    base = np.arange(60, dtype=np.float64)
    scans = [base.reshape(-1, 3), base.astype(np.float32).reshape(-1, 6)[:, :3],
             base.astype(np.float32), base.tolist()]
    arr, m, keep = capi.scan_array(scans, np.zeros((4, 6)))
    assert [k.shape for k in keep] == [(20, 3), (10, 3), (20, 3), (20, 3)]
    assert all(k.dtype == np.float32 and k.flags.c_contiguous for k in keep)
    assert [s.xyz for s in arr] == [k.ctypes.data for k in keep]


def test_refused():
    one = np.zeros((1, 3), np.float32)
    with pytest.raises(IndexError):
        capi.scan_array([one], np.zeros((1, 5)))
    # fewer poses than scans: the rest stays empty, and the C side refuses it
    arr, m, _ = capi.scan_array([one, one], np.zeros((1, 6)))
    assert m == 2 and arr[1].xyz is None
    assert capi.scan_array([], [])[1] == 0
