"""Poses as tensors, taken element by element where NumPy does not read them as an array."""
import numpy as np
import torch

from cuda_ndt_matcher_gb300 import capi


class Remote:
    """A row whose elements are numbers but which refuses to become an array (as a tensor on a GPU)."""

    def __init__(self, row):
        self.row = row

    def __len__(self):
        return len(self.row)

    def __getitem__(self, k):
        return self.row[k]

    def __array__(self, *a, **k):
        raise TypeError("not convertible")


def test_rows_that_numpy_refuses():
    scans = [np.zeros((2, 3), np.float32)] * 2
    p = np.arange(12.0).reshape(2, 6)
    for poses in (torch.tensor(p, requires_grad=True), list(torch.tensor(p, requires_grad=True)),
                  [Remote(r) for r in p], list(torch.tensor(p))):
        arr, m, _ = capi.scan_array(scans, poses)
        assert m == 2
        assert [list(s.initial_pose) for s in arr] == p.tolist()
