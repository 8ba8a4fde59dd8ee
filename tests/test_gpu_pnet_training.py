"""The training kernels at the sizes where their tiles change: gradients against the FP64
restatement, the tcgen05 GEMM's tile shapes against torch, and whole training steps (sampling,
features, forward, backward, Adam) against a NumPy restatement fed with the gradients."""
import numpy as np
import pytest

from cuda_ndt_matcher_gb300 import capi, synth

pytestmark = pytest.mark.gpu


# tiles of 256 x 256 (from 96 of them), 128 x 128 (from 152), the deep ring (K beyond 2,048 with few
# tiles), 128 x 64; ragged edges of each
@pytest.mark.parametrize("m,n,k,splits", [
    (2560, 2560, 128, 1), (2500, 2504, 192, 1), (2304, 2600, 64, 1),
    (1600, 1540, 320, 1), (300, 520, 4096, 16), (130, 72, 2112, 1), (100, 200, 2176, 1),
    (640, 512, 1536, 16), (129, 65 * 4, 64, 1), (1, 4, 64, 1)])
def test_gemm_tiles(gpu, m, n, k, splits):
    import torch
    g = torch.Generator(device="cpu").manual_seed(m + n + k)
    a = torch.randn(m, k, generator=g).to(torch.bfloat16).cuda()
    b = torch.randn(n, k, generator=g).to(torch.bfloat16).cuda()
    ref = a.double() @ b.double().T
    d = capi.gemm_bf16(a, b, splits).double()
    # products are exact, K f32 additions of terms whose sum of magnitudes is |a| |b|
    bound = (k + splits) * 2.0 ** -23 * (a.double().abs() @ b.double().abs().T)
    assert bool(((d - ref).abs() <= bound).all())


@pytest.mark.parametrize("cfg,b", [
    (dict(input_dim=4928, hidden=512, hidden_layers=1, proposals=16, batch=192), 192),
    (dict(input_dim=8256, hidden=576, hidden_layers=2, proposals=32, batch=64), 64),
    (dict(input_dim=192, hidden=192, hidden_layers=3, proposals=48, batch=320), 320)], ids=str)
def test_gradients(gpu, cfg, b):
    """Weight gradients of 128 x 128 tiles with an odd multiple of 64 columns, and of 64."""
    from oracle import pnet_oracle as O
    net = capi.PNet(seed=3, **cfg)
    dims = [cfg["input_dim"]] + [cfg["hidden"]] * cfg["hidden_layers"] + [4 * cfg["proposals"]]
    rng = np.random.default_rng(1)
    x = (rng.uniform(0, 1, (b, dims[0])) < 0.1).astype(np.float32)
    T = np.stack([rng.uniform(-5, 5, b), rng.uniform(-5, 5, b), rng.uniform(-np.pi, np.pi, b)],
                 1).astype(np.float32)
    loss, g = net.debug_grad(x, T)
    Lr, gr = O.forward_backward(net.params(), dims, x.astype(np.float64), T.astype(np.float64),
                                cfg["proposals"])
    assert abs(loss - Lr) <= 1e-3 * abs(Lr)
    off = 0
    for i, o in zip(dims[:-1], dims[1:]):
        for n in (i * o, o):  # W then b; the bound is the network's own gradient test's
            a, r = g[off:off + n], gr[off:off + n]
            assert np.linalg.norm(a - r) <= 2e-2 * np.linalg.norm(r) + 1e-7, (off, n)
            off += n
    net.close()


M64 = (1 << 64) - 1


def sm64(s):
    s[0] = (s[0] + 0x9e3779b97f4a7c15) & M64
    z = s[0]
    z = ((z ^ (z >> 30)) * 0xbf58476d1ce4e5b9) & M64
    z = ((z ^ (z >> 27)) * 0x94d049bb133111eb) & M64
    return z ^ (z >> 31)


def batch_of(seed, step, B, scans, poses, img, ox, oy, rng_xy=5.0):
    """Features and targets of a training step, from the definitions, in float32."""
    f = np.float32
    X = np.zeros((B, 36864), f)
    T = np.zeros((B, 3), f)
    unit = lambda s: f(sm64(s) >> 40) * f(2.0 ** -24)
    for b in range(B):
        s = [(seed ^ (0x9e3779b97f4a7c15 * (step + 1)) ^ (0xd1b54a32d192ed03 * (b + 1))) & M64]
        sm64(s)
        k = sm64(s) % len(scans)
        ex, ey = ((f(2) * unit(s) - f(1)) * f(rng_xy) for _ in range(2))
        yaw = (f(2) * unit(s) - f(1)) * f(np.pi)
        c = poses[k]
        cx, cy, cz = f(c[0]) + ex, f(c[1]) + ey, f(c[2])
        dy = float(f(c[5]) - yaw)
        T[b] = -ex, -ey, dy - 2 * np.pi * np.floor((dy + np.pi) / (2 * np.pi))
        co, si = f(np.cos(yaw)), f(np.sin(yaw))
        p = scans[k]
        g = np.floor(np.stack([co * p[:, 0] - si * p[:, 1] + f(32),
                               si * p[:, 0] + co * p[:, 1] + f(32), p[:, 2] + f(2)], 1)).astype(int)
        g = g[((g >= 0) & (g < [64, 64, 8])).all(1)]
        X[b, (g[:, 0] * 64 + g[:, 1]) * 8 + g[:, 2]] = 1
        i = np.arange(64, dtype=f)
        ix = np.floor(cx - f(32) + i + f(0.5) - f(ox)).astype(int)
        iy = np.floor(cy - f(32) + i + f(0.5) - f(oy)).astype(int)
        ok = ((ix >= 0) & (ix < img.shape[0]))[:, None] & ((iy >= 0) & (iy < img.shape[1]))
        h = img[np.clip(ix, 0, img.shape[0] - 1)[:, None], np.clip(iy, 0, img.shape[1] - 1)]
        v = f(0.1) + np.clip((h - cz + f(2)) / f(10), f(0), f(0.9))
        X[b, 32768:] = np.where(ok & np.isfinite(h), v, 0).ravel()
    return X, T


def test_training_steps(gpu):
    """Three steps: the weights move as Adam with the gradients of the restated batches says.
    A point within rounding of a cell's edge may fall on its other side (about one in 1e5), which
    shifts small gradients and with them an update's sign: at most 2% of the weights may be off by
    more than a tenth of a step. A misplaced tile or row is off in most of its weights."""
    B, seed, lr = 64, 5, 3e-4
    w = synth.search_queries(seed=31, n_queries=5)
    net = capi.PNet(batch=B, train_batch=B, seed=seed)
    twin = capi.PNet(batch=B, train_batch=B, seed=seed)
    mid = net.add_map(w.map_points)
    for s, t in zip(w.scans, w.true_poses):
        net.add_scan(mid, s, t)
    pts = np.asarray(w.map_points, np.float32)
    ox, oy = np.floor(pts[:, 0].min()), np.floor(pts[:, 1].min())
    cx = np.floor(pts[:, 0] - ox).astype(int)
    cy = np.floor(pts[:, 1] - oy).astype(int)
    img = np.full((cx.max() + 1, cy.max() + 1), -np.inf, np.float32)
    np.maximum.at(img, (cx, cy), pts[:, 2])
    p = net.params()
    m = np.zeros_like(p)
    v = np.zeros_like(p)
    for step in range(3):
        X, T = batch_of(seed, step, B, [np.asarray(s) for s in w.scans], w.true_poses, img, ox, oy)
        twin.set_params(p)
        g = twin.debug_grad(X, T)[1]
        m = np.float32(0.9) * m + np.float32(0.1) * g
        v = np.float32(0.999) * v + np.float32(1 - 0.999) * g * g
        want = p - lr / (1 - 0.9 ** (step + 1)) * m / (np.sqrt(v / (1 - 0.999 ** (step + 1))) + 1e-8)
        net.train(1, record_loss=False)
        p = net.params()
        off = np.abs(p - want) > 0.1 * lr
        n = 36864 * 512
        assert off[:n].mean() <= 0.02 and off[n:].mean() <= 0.02, (step, off[:n].mean())
        assert np.abs(p - want).max() <= 2.2 * lr * (step + 1)
