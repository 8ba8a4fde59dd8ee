"""Workspaces of the standalone sort and segment entry points: their sizes (a caller may have kept one
from an earlier build of the library) and the alignment they need."""
import ctypes as C

import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi


def up(x):
    return (x + 255) // 256 * 256


@pytest.mark.parametrize("n", [1, 4096, 31 * 4096, 32 * 4096, 10**6, 10**8])
def test_sizes(n):
    tiles = -(-n // 4096)
    L = capi.load()
    tb = C.c_uint64(0)
    one = C.c_void_p(16)  # not read by a size query
    assert L.ndt_detect_segments(one, n, one, one, one, None, C.byref(tb), None) == 0
    assert tb.value == 2 * up(4 * n + 4) + up(4 * tiles + 4)
    assert L.ndt_radix_sort_pairs_u64_u32(one, one, n, 0, 64, None, C.byref(tb), None) == 0
    assert tb.value == up(8 * n) + up(4 * n) + up(1024 * tiles) + up(4 * (-(-tiles // 16)) + 4)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [5, 4097, 300_000])
def test_segments_in_a_workspace_on_a_4_byte_boundary(gpu, n):
    import torch
    rng = np.random.default_rng(n)
    codes = np.sort(rng.integers(0, n // 2 + 1, n).astype(np.uint64))
    L = capi.load()
    k = torch.from_numpy(codes.view(np.int64)).cuda()
    ids, starts = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2))
    num = torch.zeros(1, dtype=torch.int32, device="cuda")
    tb = C.c_uint64(0)
    ptr = [C.c_void_p(t.data_ptr()) for t in (ids, starts, num)]
    capi.check(L.ndt_detect_segments(C.c_void_p(k.data_ptr()), n, *ptr, None, C.byref(tb), None))
    tmp = torch.empty(int(tb.value) + 4, dtype=torch.uint8, device="cuda")
    capi.check(L.ndt_detect_segments(C.c_void_p(k.data_ptr()), n, *ptr,
                                     C.c_void_p(tmp.data_ptr() + 4), C.byref(tb), None))
    torch.cuda.synchronize()
    head = np.concatenate([[True], codes[1:] != codes[:-1]])
    assert int(num.item()) == head.sum()
    np.testing.assert_array_equal(ids.cpu().numpy(), np.cumsum(head) - 1)
    np.testing.assert_array_equal(starts.cpu().numpy()[:head.sum()], np.flatnonzero(head))
