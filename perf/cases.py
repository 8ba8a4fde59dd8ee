"""The work that a user of this library has it do, as cases to be timed and checked.

A case is a dict of plain values. Its "kind" names the entry point: one scan aligned, a batch
of scans, a particle search, NVTL at many poses, a map built, a window of map tiles moved, the
proposal network trained or asked. Maps are seeded street scenes (ground, box buildings, poles,
tree blobs at the densities of synth.Sequence); scans are voxel-filtered samples of the map's
surface around a pose, in the filter's cell order, with range noise. Everything is drawn from
the seed, on the GPU.

Alignments start where a tracker's prediction does and cap their iterations below the
library's default of 30: a Newton trajectory that crosses indefinite Hessians amplifies a
last-bit difference tenfold an iteration, so the ends of a batch of 30-iteration trajectories
compare nothing. A tracker that must answer within the scan period caps them too.
"""
import ctypes as C
import math

import numpy as np
import torch

from cuda_ndt_matcher_gb300 import capi

RES = 2.0          # voxel size of the localisation maps (the library's default)
SCAN_RADIUS = 60.0
GUESS_XY, GUESS_YAW = 0.05, math.radians(0.25)  # 1 sigma of a tracker's prediction
PARTICLE_SEED = 17


def listed():
    return [
        # a live tracker's scan: 32 rings filtered at 1 m, on the 100 m map, host array in and
        # result out: the smallest call, where launches and the Newton step's latency count
        {"name": "scan_1500", "kind": "scan", "points": 1500, "map_points": 200_000,
         "extent": 100.0, "semantics": 0, "line_search": 0, "max_iterations": 10},
        # the same with a 128-ring scan on a city tile
        {"name": "scan_20k", "kind": "scan", "points": 20_000, "map_points": 5_000_000,
         "extent": 400.0, "semantics": 0, "line_search": 0, "max_iterations": 10},
        # the matcher's other Newton rule (use_gpu = false semantics: all 27 neighbours)
        {"name": "scan_cpu_rule", "kind": "scan", "points": 5003, "map_points": 1_000_000,
         "extent": 200.0, "semantics": 1, "line_search": 0, "max_iterations": 8},
        # a queue of scans of uneven size (log-uniform 2k-40k points) aligned in one call
        {"name": "queue_64", "kind": "batch", "scans": 64, "lo": 2000, "hi": 40_000,
         "map_points": 200_000, "extent": 100.0, "work_queue": 0, "cuda_graph": 1,
         "max_iterations": 5},
        # offline re-localisation of a drive: 256 scans of 20k points a call, on the form the
        # autotuner picks for them
        {"name": "batch_256", "kind": "batch", "scans": 256, "lo": 20_000, "hi": 20_000,
         "map_points": 5_000_000, "extent": 400.0, "work_queue": 8, "cuda_graph": 0,
         "max_iterations": 5},
        # initial pose after a restart: particles around a rough fix with a known heading
        {"name": "search_16x200", "kind": "search", "queries": 16, "particles": 200,
         "xy_range": 0.5, "yaw_range": 0.05, "points": 3200, "map_points": 200_000,
         "extent": 100.0, "max_iterations": 6},
        # how well a scan fits at many poses (the pose covariance estimate, a score map)
        {"name": "nvtl_20k_x_100", "kind": "nvtl", "points": 20_000, "poses": 100,
         "map_points": 5_000_000, "extent": 400.0},
        # a city tile becomes the target and the next scan's neighbours and fit are asked for
        {"name": "map_5m", "kind": "map", "map_points": 5_000_000, "extent": 400.0,
         "resolution": 2.0, "points": 20_000},
        # the same for a 2 x 2 km map with outliers
        {"name": "map_50m", "kind": "map", "map_points": 50_000_000, "extent": 2000.0,
         "resolution": 2.0, "points": 20_000},
        # a 5 x 5 window of 100 m tiles moves on: one tile out, one in, the map merged
        {"name": "tiles_25", "kind": "tiles", "tile_points": 126_000, "side": 5,
         "tile_m": 100.0, "points": 5000},
        # the proposal network trained between checkpoints, and its parameters taken out
        {"name": "train_50", "kind": "train", "steps": 50, "train_batch": 1024,
         "points": 3200, "scans": 96},
        # proposals for a full inference batch of scans
        {"name": "propose_256", "kind": "propose", "queries": 256, "points": 3200},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _extent(map_points):
    # the density of the 5M-point, 400 m tile
    return round(400.0 * math.sqrt(map_points / 5e6), 1) if map_points > 200_000 else 100.0


def draw(rng):
    kind = rng.choice(["scan", "scan", "batch", "batch", "search", "nvtl", "map", "map",
                       "tiles", "train", "propose"])
    if kind == "scan":
        m = _log(rng, 200_000, 5_000_000)
        sem = rng.choice([0, 0, 0, 1])
        return {"kind": kind, "points": _log(rng, 700, 40_000), "map_points": m,
                "extent": _extent(m), "semantics": sem,
                "line_search": 0 if sem else rng.choice([0, 0, 0, 1]),
                "max_iterations": rng.randint(5, 10)}
    if kind == "batch":
        m = _log(rng, 200_000, 5_000_000)
        lo = _log(rng, 1500, 20_000)
        hi = rng.choice([lo, min(40_000, lo * rng.randint(2, 12))])
        return {"kind": kind, "scans": _log(rng, 4, max(8, min(256, 4_000_000 // hi))),
                "lo": lo, "hi": hi, "map_points": m, "extent": _extent(m), "work_queue": rng.choice([0, 0, 4, 8]),
                "cuda_graph": rng.choice([0, 1]), "max_iterations": rng.randint(3, 5)}
    if kind == "search":
        return {"kind": kind, "queries": rng.randint(1, 16), "particles": _log(rng, 20, 200),
                "xy_range": 0.5, "yaw_range": 0.05, "points": _log(rng, 1000, 3200),
                "map_points": 200_000, "extent": 100.0, "max_iterations": rng.randint(4, 6)}
    if kind == "nvtl":
        m = _log(rng, 200_000, 5_000_000)
        return {"kind": kind, "points": _log(rng, 1000, 40_000), "poses": _log(rng, 1, 200),
                "map_points": m, "extent": _extent(m)}
    if kind == "map":
        m = _log(rng, 200_000, 20_000_000)
        return {"kind": kind, "map_points": m, "extent": _extent(m),
                "resolution": rng.choice([1.0, 2.0, 2.0, 3.0]), "points": _log(rng, 1000, 20_000)}
    if kind == "tiles":
        return {"kind": kind, "tile_points": _log(rng, 20_000, 200_000), "side": rng.randint(3, 5),
                "tile_m": 100.0, "points": _log(rng, 1000, 20_000)}
    if kind == "train":
        return {"kind": kind, "steps": rng.randint(10, 50),
                "train_batch": 64 * _log(rng, 4, 16), "points": _log(rng, 1000, 3200),
                "scans": rng.randint(32, 96)}
    return {"kind": kind, "queries": _log(rng, 1, 256), "points": _log(rng, 1000, 3200)}


# ---- inputs -----------------------------------------------------------------------------

def _gen(seed, what):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1_000_003 + what * 7919 + 12345) & 0x7FFFFFFFFFFF)
    return g


def _u(g, lo, hi, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float32) * (hi - lo) + lo


def _n(g, sigma, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32) * sigma


def _scene(n, extent, g, outliers=0.0):
    """n points of a seeded street scene over [-extent/2, extent/2]^2, in random order."""
    half, area = extent / 2, (extent / 400.0) ** 2
    nb, npole, nt = max(12, int(250 * area)), max(40, int(800 * area)), int(300 * area)
    n_out = int(n * outliers)
    n_tree = int(0.05 * n) if nt else 0
    n_pole = int(0.04 * n)
    n_wall = int(0.41 * n)
    n_ground = n - n_out - n_tree - n_pole - n_wall
    parts = []
    p = torch.empty(n_ground, 3, device="cuda")
    p[:, :2] = _u(g, -half, half, n_ground, 2)
    p[:, 2] = _n(g, 0.03, n_ground)
    parts.append(p)
    cen = _u(g, -half + 15, half - 15, nb, 2)
    side = _u(g, 8.0, 30.0, nb, 2) * (0.5 if extent <= 100.0 else 1.0)
    height = _u(g, 5.0, 20.0, nb)
    area_w = (side[:, 0] + side[:, 1]) * height
    edge = torch.cumsum(area_w.double(), 0)
    i = torch.searchsorted(edge, _u(g, 0.0, 1.0, n_wall).double() * edge[-1]).clamp(max=nb - 1)
    s, u = side[i], _u(g, -0.5, 0.5, n_wall)
    along_x = _u(g, 0.0, 1.0, n_wall) * (s[:, 0] + s[:, 1]) < s[:, 0]
    sign = torch.where(_u(g, 0.0, 1.0, n_wall) < 0.5, -0.5, 0.5)
    p = torch.empty(n_wall, 3, device="cuda")
    p[:, 0] = cen[i, 0] + torch.where(along_x, u, sign) * s[:, 0]
    p[:, 1] = cen[i, 1] + torch.where(along_x, sign, u) * s[:, 1]
    p[:, 2] = _u(g, 0.0, 1.0, n_wall) * height[i]
    parts.append(p)
    i = torch.randint(npole, (n_pole,), generator=g, device="cuda")
    cen, a = _u(g, -half, half, npole, 2), _u(g, -math.pi, math.pi, n_pole)
    p = torch.empty(n_pole, 3, device="cuda")
    p[:, 0] = cen[i, 0] + 0.15 * torch.cos(a)
    p[:, 1] = cen[i, 1] + 0.15 * torch.sin(a)
    p[:, 2] = _u(g, 0.0, 6.0, n_pole)
    parts.append(p)
    if n_tree:
        i = torch.randint(nt, (n_tree,), generator=g, device="cuda")
        cen, sig = _u(g, -half, half, nt, 2), _u(g, 1.0, 3.0, nt, 3)
        p = _n(g, 1.0, n_tree, 3) * sig[i]
        p[:, :2] += cen[i]
        p[:, 2] += 5.0
        parts.append(p)
    if n_out:
        p = _u(g, -half, half, n_out, 3)
        p[:, 2] = _u(g, -5.0, 30.0, n_out)
        parts.append(p)
    pts = torch.cat(parts)
    return pts[torch.randperm(n, generator=g, device="cuda")].contiguous()


def _poses(m, extent, g):
    """m sensor poses [m, 6]: inside the map, 1.8 m up, any heading."""
    half = max(5.0, extent / 2 - (25.0 if extent <= 100.0 else 45.0))
    p = torch.zeros(m, 6, device="cuda", dtype=torch.float64)
    p[:, :2] = _u(g, -half, half, m, 2).double()
    p[:, 2] = 1.8
    p[:, 5] = _u(g, -math.pi, math.pi, m).double()
    return p.cpu().numpy()


def _scan(points, pose, n, g):
    """n points of the map within SCAN_RADIUS of the pose, in the sensor frame, with noise."""
    d = points[:, :2] - torch.tensor(pose[:2], device="cuda", dtype=torch.float32)
    near = torch.nonzero((d * d).sum(1) < SCAN_RADIUS * SCAN_RADIUS).squeeze(1)
    q = points[near[torch.randint(len(near), (n,), generator=g, device="cuda")]].double()
    q = q - torch.tensor(pose[:3], device="cuda", dtype=torch.float64)
    c, s = math.cos(pose[5]), math.sin(pose[5])
    q = torch.stack([c * q[:, 0] + s * q[:, 1], -s * q[:, 0] + c * q[:, 1], q[:, 2]], 1).float()
    q += _n(g, 0.02, n, 3)
    cell = torch.floor(q).long() + 128
    return q[torch.argsort((cell[:, 0] * 256 + cell[:, 1]) * 256 + cell[:, 2])].contiguous()


def _guesses(true, g, xy, yaw):
    """Predictions of the true poses: N(0, xy) metres and N(0, yaw) radians off."""
    r = true.copy()
    r[:, :2] += _n(g, xy, len(true), 2).double().cpu().numpy()
    r[:, 5] += _n(g, yaw, len(true)).double().cpu().numpy()
    return r


def _scan_array(scans, poses):
    arr = (capi.Scan * len(scans))()
    for i, (s, p) in enumerate(zip(scans, poses)):
        arr[i].xyz = s.ctypes.data
        arr[i].num_points = len(s)
        for k in range(6):
            arr[i].initial_pose[k] = float(p[k])
    return arr


_RESULT = np.dtype({"names": ["pose", "score", "transform_probability", "nvtl", "hessian",
                              "converged", "iterations", "num_correspondences",
                              "oscillation_count", "status"],
                    "formats": [("f8", 6), "f8", "f8", "f8", ("f8", (6, 6)), "i4", "i4", "i4",
                                "i4", "i4"],
                    "offsets": [0, 48, 56, 64, 72, 360, 364, 368, 372, 376],
                    "itemsize": C.sizeof(capi.Result)})


def _target(case, g, **cfg):
    pts = _scene(case["map_points"], case["extent"], g)
    ctx = capi.Context(resolution=RES, **cfg)
    torch.cuda.synchronize()
    ctx.set_target_device(pts.data_ptr(), len(pts))
    return pts, ctx


def prepare(case, seed):
    g = _gen(seed, 1)
    st = {"case": case}
    kind = case["kind"]
    if kind == "scan":
        pts, ctx = _target(case, g, semantics=case["semantics"],
                           use_line_search=case["line_search"],
                           max_iterations=case["max_iterations"])
        true = _poses(1, case["extent"], g)
        st.update(ctx=ctx, scan=_scan(pts, true[0], case["points"], g).cpu().numpy(),
                  guess=_guesses(true, g, GUESS_XY, GUESS_YAW)[0], map=pts)
    elif kind == "batch":
        pts, ctx = _target(case, g, work_queue=case["work_queue"], cuda_graph=case["cuda_graph"],
                           max_iterations=case["max_iterations"])
        m = case["scans"]
        true = _poses(m, case["extent"], g)
        size = torch.exp(_u(g, math.log(case["lo"]), math.log(case["hi"]), m)).round().long()
        scans = [_scan(pts, true[i], n, g).cpu().numpy() for i, n in enumerate(size.tolist())]
        guess = _guesses(true, g, GUESS_XY, GUESS_YAW)
        st.update(ctx=ctx, scans=scans, guess=guess, arr=_scan_array(scans, guess),
                  res=(capi.Result * m)(), map=pts)
    elif kind == "search":
        pts, ctx = _target(case, g, max_iterations=case["max_iterations"])
        true = _poses(case["queries"], case["extent"], g)
        st.update(ctx=ctx, scans=[_scan(pts, t, case["points"], g).cpu().numpy() for t in true],
                  prior=_guesses(true, g, GUESS_XY, GUESS_YAW), map=pts)
    elif kind == "nvtl":
        pts, ctx = _target(case, g)
        true = _poses(1, case["extent"], g)
        at = _guesses(np.repeat(true, case["poses"], 0), g, 0.3, math.radians(1.0))
        st.update(ctx=ctx, scan=_scan(pts, true[0], case["points"], g).cpu().numpy(),
                  T=np.stack([_rz(p) for p in at]), map=pts)
    elif kind == "map":
        pts = _scene(case["map_points"], case["extent"], g,
                     0.05 if case["map_points"] > 5_000_000 else 0.0)
        true = _poses(1, case["extent"], g)
        st.update(ctx=capi.Context(resolution=case["resolution"]), map=pts,
                  scan=_scan(pts, true[0], case["points"], g).cpu().numpy(), T=_rz(true[0])[None])
        torch.cuda.synchronize()
    elif kind == "tiles":
        side, size, tp = case["side"], case["tile_m"], case["tile_points"]
        ext = size * (side + 1)
        pts = _scene(tp * side * (side + 1), ext, g)
        # the scene's own square, cut in columns (x) and rows (y) of tiles; one column more than
        # the window holds, which moves back and forth over its middle row's ends
        ix = torch.clamp(((pts[:, 0] + ext / 2) / size).long(), 0, side)
        iy = torch.clamp(((pts[:, 1] + ext / 2) / size).long(), 0, side)
        tiles = {(x, y): pts[(ix == x) & (iy == y)].cpu().numpy()
                 for x in range(side + 1) for y in range(side)}
        ctx = capi.Context(resolution=RES)
        for x in range(side):
            for y in range(side):
                ctx.tile_put(x * 16 + y, tiles[(x, y)])
        ctx.tiles_commit()
        mid = side // 2
        true = np.array([[size - ext / 2, -size / 2, 1.8, 0.0, 0.0, 0.3]])  # beside the left end
        st.update(ctx=ctx, ends=[(0, mid), (side, mid)], tiles=tiles, at=0, map=pts,
                  scan=_scan(pts, true[0], case["points"], g).cpu().numpy(), T=_rz(true[0])[None])
    elif kind in ("train", "propose"):
        pts = _scene(1_250_000, 200.0, g)
        n = case["scans"] if kind == "train" else case["queries"]
        true = _poses(n, 200.0, g)
        scans = [_scan(pts, t, case["points"], g).cpu().numpy() for t in true]
        cfg = {"train_batch": case["train_batch"]} if kind == "train" else {}
        net = capi.PNet(seed=(int(seed) & 0xFFFF) + 1, **cfg)
        mid = net.add_map(pts.cpu().numpy())
        st.update(net=net, map_id=mid, scans=scans)
        if kind == "train":
            for s, t in zip(scans, true):
                net.add_scan(mid, s, t)
        else:
            coarse = true + 0.0
            coarse[:, :2] += _u(g, -5.0, 5.0, n, 2).double().cpu().numpy()
            coarse[:, 5] = _u(g, -math.pi, math.pi, n).double().cpu().numpy()
            st.update(coarse=coarse)
    else:
        raise ValueError(kind)
    return st


def _rz(p):
    """Row-major 3 x 4 transform of a pose whose roll and pitch are zero."""
    c, s = math.cos(p[5]), math.sin(p[5])
    return np.array([c, -s, 0, p[0], s, c, 0, p[1], 0, 0, 1, p[2]], np.float64)


# ---- one pass ---------------------------------------------------------------------------

def run(st):
    kind = st["case"]["kind"]
    if kind == "scan":
        return st["ctx"].align(st["scan"], st["guess"])
    if kind == "batch":
        st["ctx"].align_batch_raw(st["arr"], st["res"])
        r = np.frombuffer(st["res"], _RESULT)
        return {k: r[k] for k in _RESULT.names}
    if kind == "search":
        c = st["case"]
        est = st["ctx"].initial_pose_search(st["scans"], st["prior"],
                                            num_particles=c["particles"], xy_range=c["xy_range"],
                                            yaw_range=c["yaw_range"], seed=PARTICLE_SEED)
        return {k: np.array([e[k] for e in est]) for k in est[0]}
    if kind == "nvtl":
        nvtl, tp = st["ctx"].eval_batch(st["scan"], st["T"])
        return {"nvtl": nvtl, "tp": tp}
    if kind == "map":
        st["ctx"].set_target_device(st["map"].data_ptr(), len(st["map"]))
        return _ask(st)
    if kind == "tiles":
        # the tile behind leaves, the tile ahead comes in; the next pass moves back
        ctx, a = st["ctx"], st["at"]
        out, into = st["ends"][a], st["ends"][1 - a]
        st["at"] = 1 - a
        ctx.tile_remove(out[0] * 16 + out[1])
        ctx.tile_put(into[0] * 16 + into[1], st["tiles"][into])
        ctx.tiles_commit()
        return _ask(st)
    if kind == "train":
        st["net"].train(st["case"]["steps"], record_loss=False)
        return {"params": st["net"].params()}
    poses, logits = st["net"].propose(st["map_id"], st["scans"], st["coarse"])
    return {"poses": poses, "logits": logits}


def _ask(st):
    """What a program takes from a new map: its description, and the next scan's neighbours
    and fit at the predicted pose."""
    ctx = st["ctx"]
    i = ctx.map_info()
    nvtl, tp = ctx.eval_batch(st["scan"], st["T"])
    T = st["T"][0].reshape(3, 4)
    idx, cnt = ctx.neighbors((st["scan"] @ T[:, :3].T.astype(np.float32)
                              + T[:, 3].astype(np.float32)))
    return {"nvtl": nvtl, "tp": tp, "idx": idx, "cnt": cnt,
            "info": np.array([i.num_points, i.num_segments, i.num_voxels, i.hash_capacity]
                             + list(i.min_coord) + list(i.max_coord), np.int64)}


# ---- what a pass cannot do without ------------------------------------------------------

def work(case):
    """Points once in, results once out. Arithmetic: a point's transform and contraction cost
    165 operations an iteration and a point-voxel pair 65, with about five pairs a point and
    five iterations an alignment."""
    kind = case["kind"]
    per_point = 165 + 5 * 65
    if kind in ("scan", "batch", "search"):
        if kind == "scan":
            jobs, pts = 1, case["points"]
            read = pts
        elif kind == "batch":
            jobs = case["scans"]
            lo, hi = case["lo"], case["hi"]
            read = jobs * (lo if hi == lo else (hi - lo) / math.log(hi / lo))
            pts = read
        else:
            jobs = case["queries"] * case["particles"]
            read = case["queries"] * case["points"]
            pts = jobs * case["points"]
        return {"bytes": 12 * read + 400 * jobs, "flops": 5 * per_point * pts}
    if kind == "nvtl":
        return {"bytes": 12 * case["points"] + 112 * case["poses"],
                "flops": case["points"] * case["poses"] * (30 + 5 * 40)}
    if kind == "map":
        # the points, then a centroid and an inverse covariance for each voxel
        return {"bytes": 12 * case["map_points"] + 36 * 0.03 * case["map_points"]
                + 48 * case["points"], "flops": 30 * case["map_points"]}
    if kind == "tiles":
        n = case["tile_points"]
        return {"bytes": 12 * n + 88 * 0.03 * n * case["side"] ** 2 + 48 * case["points"],
                "flops": 30 * n}
    w = 36864 * 512 + 3 * 512 * 512 + 512 * 64
    if kind == "train":
        b = case["train_batch"]
        # forward and both gradients (none for the input), Adam's state once each way
        return {"bytes": case["steps"] * (w * 26 + 2.0 * b * 36864),
                "flops": case["steps"] * (4.0 * b * w + 2.0 * b * (w - 36864 * 512))}
    n = case["queries"]
    return {"bytes": 2.0 * w + 12.0 * n * case["points"] + n * 16 * 56, "flops": 2.0 * n * w}


# ---- the same in 64 bits ----------------------------------------------------------------

def exact(case, seed):
    """Alignments, scores and NVTL in 64 bits from the same f32 points; None for line search,
    the particle search (thousands of alignments), the moved tiles (their map depends on the
    passes so far), whole numbers and the bf16 network."""
    kind = case["kind"]
    if kind in ("train", "propose", "search", "tiles") or case.get("line_search"):
        return None
    st = prepare(case, seed)
    res = case.get("resolution", RES)
    if kind in ("nvtl", "map"):
        v = _Voxels(st["map"], res, near=st["T"][0][[3, 7]] if kind == "map" else None)
        s = torch.tensor(st["scan"], device="cuda").double()
        got = [v.score(s, torch.tensor(t.reshape(3, 4), device="cuda")) for t in st["T"]]
        out = {"nvtl": np.array([g[0] for g in got]), "tp": np.array([g[1] for g in got])}
        return out if kind == "nvtl" else dict(out, idx=None, cnt=None, info=None)
    v = _Voxels(st["map"], res)
    sem = case.get("semantics", 0)
    scans = [st["scan"]] if kind == "scan" else st["scans"]
    guess = [st["guess"]] if kind == "scan" else st["guess"]
    got = [v.align(torch.tensor(s, device="cuda").double(), p, sem, case["max_iterations"])
           for s, p in zip(scans, guess)]
    keys = ("pose", "score", "transform_probability", "nvtl", "hessian")
    out = {k: np.stack([np.asarray(g[k]) for g in got]) for k in keys}
    if kind == "scan":
        out = {k: (x[0] if x[0].ndim else float(x[0])) for k, x in out.items()}
    return out


class _Voxels:
    """The voxel map and the NDT score, gradient and Hessian, in 64 bits."""

    def __init__(self, pts, res, near=None):
        if near is not None:  # only the cells that a scan there can reach
            d = pts[:, :2] - torch.tensor(near, device="cuda", dtype=torch.float32)
            pts = pts[(d * d).sum(1) < (SCAN_RADIUS + 6 * res) ** 2]
        self.res = res
        cell = torch.floor(pts / res).long()
        self.lo = cell.amin(0) - 2
        self.dim = cell.amax(0) - self.lo + 3
        key = self._key(cell)
        self.keys, inv, cnt = torch.unique(key, return_inverse=True, return_counts=True)
        n, p = len(self.keys), pts.double()
        mean = torch.zeros(n, 3, dtype=torch.float64, device="cuda").index_add_(0, inv, p)
        mean /= cnt[:, None]
        c = p - mean[inv]
        cov = torch.zeros(n, 9, dtype=torch.float64, device="cuda")
        cov.index_add_(0, inv, (c[:, :, None] * c[:, None, :]).reshape(-1, 9))
        ok = cnt >= 6
        cov = cov.reshape(-1, 3, 3)[ok] / (cnt[ok] - 1)[:, None, None]
        lam, vec = np.linalg.eigh(cov.cpu().numpy())
        lam = np.maximum(lam, 0.01 * lam[:, 2:])
        self.icov = torch.tensor((vec / lam[:, None, :]) @ vec.transpose(0, 2, 1), device="cuda")
        self.keys, self.mean = self.keys[ok], mean[ok]
        o = torch.arange(-1, 2, device="cuda")
        self.off = torch.cartesian_prod(o, o, o)
        c1, c2 = 10.0 * 0.45, 0.55 / float(np.float32(res)) ** 3
        d3 = -math.log(c2)
        self.d1 = -math.log(c1 + c2) - d3
        self.d2 = -2.0 * math.log((-math.log(c1 * math.exp(-0.5) + c2) - d3) / self.d1)

    def _key(self, cell):
        c = cell - self.lo
        k = (c[..., 0] * self.dim[1] + c[..., 1]) * self.dim[2] + c[..., 2]
        return torch.where(((c >= 0) & (c < self.dim)).all(-1), k, -1)

    def pairs(self, q, most):
        """(point, voxel) of the neighbours within one resolution, `most` a point in order."""
        cell = torch.floor(q / self.res).long()
        k = self._key(cell[:, None, :] + self.off)
        at = torch.searchsorted(self.keys, k).clamp(max=len(self.keys) - 1)
        hit = self.keys[at] == k
        d = q[:, None, :] - self.mean[at]
        hit &= (d * d).sum(2) <= self.res * self.res
        hit &= torch.cumsum(hit, 1) <= most
        i, j = torch.nonzero(hit, as_tuple=True)
        return i, at[i, j]

    def terms(self, q, most):
        i, v = self.pairs(q, most)
        x, Cv = q[i] - self.mean[v], self.icov[v]
        c = torch.einsum("nij,nj->ni", Cv, x)
        e = torch.exp(-0.5 * self.d2 * (x * c).sum(1))
        return i, c, Cv, e

    def score(self, s, T):
        q = s @ T[:, :3].T + T[:, 3]
        i, _, _, e = self.terms(q, 27)
        e = -self.d1 * e
        best = torch.full((len(q),), -math.inf, dtype=torch.float64, device="cuda")
        best.scatter_reduce_(0, i, e, "amax")
        best = best[torch.isfinite(best)]
        return float(best.mean()) if len(best) else 0.0, float(e.mean()) if len(e) else 0.0

    def derivatives(self, s, pose, sem):
        f = [_axis(a, t) for a, t in enumerate(pose[3:])]
        mul = lambda a, b, c: f[0][a] @ f[1][b] @ f[2][c]  # noqa: E731
        R = torch.tensor(mul(0, 0, 0), device="cuda")
        A = np.stack([mul(1, 0, 0), mul(0, 1, 0), mul(0, 0, 1)])
        B = {(0, 0): mul(2, 0, 0), (0, 1): mul(1, 1, 0), (0, 2): mul(1, 0, 1),
             (1, 1): mul(0, 2, 0), (1, 2): mul(0, 1, 1), (2, 2): mul(0, 0, 2)}
        B[(1, 1)][0, 2] = math.sin(pose[4])  # the reference's sign of this entry
        q = s @ R.T + torch.tensor(pose[:3], device="cuda")
        i, c, Cv, e = self.terms(q, 27 if sem else 8)
        keep = (self.d2 * e >= 0) & (self.d2 * e <= 1) if sem else torch.ones_like(e).bool()
        e = torch.where(keep, e, 0.0)
        w = self.d1 * self.d2 * e
        J = torch.zeros(len(s), 3, 6, dtype=torch.float64, device="cuda")
        J[:, :, :3] = torch.eye(3, device="cuda")
        J[:, :, 3:] = torch.einsum("kij,nj->nik", torch.tensor(A, device="cuda"), s)
        G = w[:, None] * c
        M = w[:, None, None] * (Cv - self.d2 * c[:, :, None] * c[:, None, :])
        Ji = J[i]
        g = torch.einsum("nik,ni->k", Ji, G).cpu().numpy()
        H = torch.einsum("nik,nij,njl->kl", Ji, M, Ji).cpu().numpy()
        GP = torch.einsum("ni,nj->ij", G, s[i]).cpu().numpy()
        for (k, l), b in B.items():
            H[3 + k, 3 + l] += (b * GP).sum()
            if k != l:
                H[3 + l, 3 + k] += (b * GP).sum()
        return float((-self.d1 * e).sum()), g, H, len(i)

    def align(self, s, pose, sem, most):
        pose = np.array(pose, np.float64)
        best, last, out = (-math.inf, pose.copy()), None, None
        eps = 0.01 if sem else float(np.float32(0.01))
        for it in range(most):
            score, g, H, n = self.derivatives(s, pose, sem)
            lam, V = np.linalg.eigh(H)
            if sem:
                if score > best[0]:
                    best = (score, pose.copy())
                last = H
                if not (lam < 0).all():
                    lam = np.where(lam > -1e-3, -1e-3, lam)
                x = V @ ((V.T @ -g) / lam)
                dn = math.sqrt(x @ x)
                if dn < eps:
                    out = (pose, score, H)
                    break
                x /= dn
                pose = pose + (x if g @ x > 0 else -x) * min(dn, 0.1)
                continue
            x = V @ ((V.T @ -g) / np.abs(lam))
            x = x if g @ x > 0 else -x
            dn = math.sqrt(x @ x)
            pose = pose + x * (min(dn, 0.1) / dn)
            if min(dn, 0.1) < eps or it + 1 == most:
                out = (pose, score, H)
                break
        if out is None:
            out = (best[1], best[0], last)
        p = out[0]
        f = [_axis(a, t)[0] for a, t in enumerate(p[3:])]
        T = np.concatenate([f[2] @ f[1] @ f[0], p[:3, None]], 1)
        return {"pose": p, "score": out[1], "transform_probability": out[1] / len(s),
                "nvtl": self.score(s, torch.tensor(T, device="cuda"))[0], "hessian": out[2]}


def _axis(a, t):
    """Rotation about axis a by t and its first two derivatives."""
    c, s = math.cos(t), math.sin(t)
    i, j = (a + 1) % 3, (a + 2) % 3
    r = np.zeros((3, 3, 3))
    for d, (u, v) in enumerate([(c, s), (-s, c), (-c, -s)]):
        r[d, i, i] = r[d, j, j] = u
        r[d, i, j], r[d, j, i] = -v, v
    r[0, a, a] = 1.0
    return r
