"""The Newton step's 6x6 solve on the definite path, from the traced Hessians, gradients and solutions of
alignments on every kernel, against a solve in extended precision."""
import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi, synth
from parity_helpers import hessian_from_trace_row

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,scans", [(0, 6), (-1, 6), (2, 6), (0, 120)])
def test_definite_solves(gpu, form, scans):
    w = synth.queue_scans(seed=67, n_scans=6, lo=2000, hi=9000)
    rng = np.random.default_rng(2)
    poses = w.true_poses[np.arange(scans) % 6].copy()
    poses[:, :2] += rng.uniform(-0.5, 0.5, (scans, 2))
    poses[:, 5] += rng.uniform(-0.05, 0.05, scans)
    ctx = capi.Context(max_iterations=12, work_queue=form)
    ctx.set_target(w.map_points)
    ctx.trace(True)
    ctx.align_batch([w.scans[i % 6] for i in range(scans)], poses)
    seen = 0
    for i in range(scans):
        for row in ctx.read_trace(i):
            if row[42] != 0:  # eigen path
                continue
            H, g, x = hessian_from_trace_row(row), row[9:15], row[36:42]
            s = 1.0 if H[0, 0] > 0 else -1.0  # H is definite: (s H) x = -g
            want = np.linalg.solve(s * H, -g).astype(np.longdouble)
            Hl = (s * H).astype(np.longdouble)
            for _ in range(4):  # refined in extended precision
                want = want + np.linalg.solve(s * H, (-g - Hl @ want).astype(float))
            # the last correction is below 1e-13 of x, and each residual is rounded in FP64
            bound = 1e-13 + 8 * np.linalg.cond(H) * 2.0**-53
            assert np.abs(x - want).max() <= bound * np.abs(want).max(), (i, row[0])
            seen += 1
    assert seen >= scans
