"""A new tile takes the buffers of the last removed one: whatever their sizes, and also when the
removed or the new tile has no finite point, the committed map is that of the resident tiles."""
import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("old,new", [(4096, 60_000), (60_000, 4097), (60_000, 60_000),
                                     (60_000, 0), (0, 60_000), (1, 30_000)])
@pytest.mark.parametrize("wait", [True, False])
def test_put_after_remove(gpu, old, new, wait):
    pts = np.ascontiguousarray(synth.Sequence(seed=7, n_map=300_000, n_scans=1).map)
    keep, a, b = pts[:150_000], pts[150_000:150_000 + old], pts[220_000:220_000 + new]
    nothing = np.full((50, 3), np.nan, np.float32)
    a, b = (x if len(x) else nothing for x in (a, b))
    ctx = capi.Context()
    ctx.tile_put(1, keep)
    ctx.tile_put(2, a)
    ctx.tile_put(3, a)
    ctx.tiles_commit(wait=True)
    ctx.tile_remove(3)   # kept for the next put
    ctx.tile_remove(2)   # kept in its place
    ctx.tile_put(4, b)   # takes it
    ctx.tile_put(5, b[: len(b) // 2 + 1])
    ctx.tiles_commit(wait=wait)
    while ctx.tiles_status()["pending"]:
        pass
    assert ctx.tiles_status()["last_rc"] == 0
    ref = capi.Context()
    ref.set_target(np.concatenate([keep, b, b[: len(b) // 2 + 1]]))
    for x, y in zip(ctx.map_voxels(), ref.map_voxels()):
        assert np.array_equal(x, y)
