"""Performance cases of the LiDAR perception path, through the package's public entry points.

A case is one call pattern of a program that uses the framework: a sensor node that hands over one
scan (`scan`), a vehicle or a log replay that hands over many (`batch`), resident scans replayed as a
captured graph (`prepared`), several sensors served as they arrive (`serve`), the outlier filter
before the pipeline (`filtered`), and the single stages by themselves (`segment`, `noise`, `cluster`,
`polygons`). Scan shapes are the ones of the synthetic workloads: 32/64/128 rings x 1024-4096 azimuth
bins, return rate 0.3-1, 10-200 obstacles, flat / sloped / undulating ground, and unorganised clouds of
up to 1M points with clutter near the sensor. Scans are ray-cast on the GPU from the seed, so another
seed is another scene.
"""
import math
import os
import sys

import numpy as np
import torch

_REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_REPO, "lidar-processing-v2_gb300"))

import lidar_gb300 as lp  # noqa: E402

SHAPES = [(r, w) for r in (32, 64, 128) for w in (1024, 2048, 4096)]
BOX = np.dtype([("corners", "<f8", (4, 2)), ("area", "<f4"), ("angle_rad", "<f4"), ("is_valid", "<i4"), ("pad", "<i4")])
assert BOX.itemsize == lp.ctypes.sizeof(lp.BoundingBox)


def listed():
    return [
        # the smallest whole call: a sparse scan of a 32-ring sensor, where latency and launches count
        {"name": "scan_small", "kind": "scan", "rings": 32, "bins": 1024, "rate": 0.3, "obstacles": 20, "ring": "given",
         "pinned": True},
        # the ordinary call: one 64 x 2048 scan in page-locked buffers, rings derived on the device
        {"name": "scan_64x2048", "kind": "scan", "rings": 64, "bins": 2048, "rate": 0.9, "obstacles": 29,
         "ring": "computed", "pinned": True},
        # the densest single scan of the configurations, in ordinary (pageable) numpy buffers
        {"name": "scan_128x4096", "kind": "scan", "rings": 128, "bins": 4096, "rate": 0.9, "obstacles": 120, "ring": "given",
         "pinned": False},
        # the six sensors of a vehicle in one call
        {"name": "batch6", "kind": "batch", "scans": 6, "ring": "given", "pinned": True},
        # the headline workload: 64 scans of uneven size in one call, host buffers in and out
        {"name": "batch64", "kind": "batch", "scans": 64, "ring": "given", "pinned": True},
        # resident scans: inputs copied again, graph replayed, results downloaded
        {"name": "prepared16", "kind": "prepared", "scans": 16},
        # a burst of the serving workload: one scan of each of six sensors submitted, all polled
        {"name": "serve6", "kind": "serve", "scans": 6},
        # the outlier filter before the pipeline, unorganised 1M-point clouds
        {"name": "filtered4x1M", "kind": "filtered", "scans": 4, "points": 1000000},
        # single stages: the filter on one ordinary cloud with its default configuration
        {"name": "noise_110k", "kind": "noise", "points": 110000, "stride": 3, "default": True},
        # ground segmentation of a cloud without rings, with the colour image
        {"name": "segment_64x2048", "kind": "segment", "rings": 64, "bins": 2048, "rate": 0.9, "obstacles": 29, "image": True},
        # clustering of one scan's obstacle points
        {"name": "cluster_40k", "kind": "cluster", "points": 40001, "stride": 4, "elevation": 3.0},
        # hull and both boxes of single clusters, 3 to 20k points each
        {"name": "polygons12", "kind": "polygons", "polygons": 12, "smallest": 3, "largest": 20000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["scan", "scan", "batch", "batch", "prepared", "serve", "filtered", "noise", "segment", "cluster",
                       "polygons"])
    c = {"kind": kind}
    if kind in ("scan", "segment"):
        c.update(rings=rng.randint(24, 128), bins=_log(rng, 900, 4096), rate=round(rng.uniform(0.3, 1.0), 3),
                 obstacles=rng.randint(10, 200))
    if kind == "segment":
        c.update(image=rng.random() < 0.5)
    elif kind == "scan":
        c.update(ring=rng.choice(["given", "computed", "none"]), pinned=rng.random() < 0.6)
    elif kind == "batch":
        c.update(scans=_log(rng, 2, 64), ring=rng.choice(["given", "computed"]), pinned=rng.random() < 0.75)
    elif kind == "prepared":
        c.update(scans=_log(rng, 1, 40))
    elif kind == "serve":
        c.update(scans=rng.randint(2, 6))
    elif kind == "filtered":
        c.update(scans=rng.randint(1, 4), points=_log(rng, 60000, 1000000))
    elif kind == "noise":
        c.update(points=_log(rng, 20000, 600000), stride=rng.choice([3, 4]), default=rng.random() < 0.5)
    elif kind == "cluster":
        c.update(points=_log(rng, 1000, 150000), stride=rng.choice([3, 4]), elevation=rng.choice([1.5, 3.0]))
    elif kind == "polygons":
        c.update(polygons=rng.randint(4, 12), smallest=3, largest=_log(rng, 200, 20000))
    return c


# ------------------------------------------------------------------ inputs
def _kept_points(rings, bins, rate):
    """Returns of a scan: `rate` of the rays that meet something (a 128-ring sensor looks up as well)."""
    return max(1, int(rings * bins * rate * (0.62 if rings > 96 else 0.88)))


def _scan(seed, rings, bins, rate, obstacles, ground, wall):
    """(xyzi N x 4 float32, ring uint16 N, segmenter configuration) of a spinning sensor 1.73 m above the ground: rays cast
    against the ground, boxes, vertical cylinders and a wall, ring by ring from the top, ascending
    azimuth; Gaussian range and height noise, dropped returns."""
    dev = "cuda"
    g = torch.Generator(device=dev).manual_seed(seed & 0x7FFFFFFF)
    up, down = (15.0, -25.0) if rings > 96 else (2.0, -24.8)
    R = rings * bins
    el = torch.linspace(math.radians(up), math.radians(down), rings, device=dev)[:, None].expand(rings, bins).reshape(1, R)
    az = ((torch.arange(bins, device=dev) + 0.5) * (2 * math.pi / bins))[None, :].expand(rings, bins).reshape(1, R)
    dx, dy, dz = torch.cos(el) * torch.cos(az), torch.cos(el) * torch.sin(az), torch.sin(el)

    def uni(n, lo, hi):
        return torch.rand(n, generator=g, device=dev) * (hi - lo) + lo

    def height(x, y):
        z = torch.full_like(x, -1.73)
        if ground == 2:
            z = z + 0.3 * torch.sin(x * (2 * math.pi / 30)) + 0.02 * torch.sin(y * (2 * math.pi / 7))
        if ground:
            z = z + math.tan(math.radians(4.0)) * torch.clamp(torch.sqrt(x * x + y * y) - 20.0, min=0.0)
        return z

    # ground: a coarse march along the ray, then bisection
    far = 80.0
    if ground == 0:
        t_ground = torch.where(dz < -1e-6, -1.73 / torch.clamp(dz, max=-1e-6), torch.full_like(dz, 1e9))
    else:
        lo, hi = torch.zeros_like(dz), torch.full_like(dz, 1e9)
        t = 0.5
        while t < far:
            s = t + max(0.25, 0.02 * t)
            crossed = (hi > 1e8) & (s * dz < height(s * dx, s * dy))
            lo, hi = torch.where(crossed, torch.full_like(lo, t), lo), torch.where(crossed, torch.full_like(hi, s), hi)
            t = s
        for _ in range(12):
            m = 0.5 * (lo + hi)
            under = m * dz < height(m * dx, m * dy)
            lo, hi = torch.where(under, lo, m), torch.where(under & (hi < 1e8), m, hi)
        t_ground = hi
    # boxes (the wall is one) and cylinders, a few at a time against every ray
    nb = obstacles * 2 // 3
    nc = obstacles - nb
    rad, ang = torch.sqrt(uni(nb + nc, 25.0, 1600.0)), uni(nb + nc, 0.0, 2 * math.pi)
    cx, cy = rad * torch.cos(ang), rad * torch.sin(ang)
    half = torch.stack([uni(nb, 0.25, 3.0), uni(nb, 0.25, 3.0)])
    tall, yaw = uni(nb, 0.5, 6.0), uni(nb, 0.0, 2 * math.pi)
    bx, by = cx[:nb], cy[:nb]
    if wall:
        a = uni(1, 0.0, 2 * math.pi)
        bx, by = torch.cat([bx, 25 * torch.cos(a)]), torch.cat([by, 25 * torch.sin(a)])
        half = torch.cat([half, torch.tensor([[15.0], [0.1]], device=dev)], 1)
        tall, yaw = torch.cat([tall, torch.full_like(a, 3.0)]), torch.cat([yaw, a + 0.5 * math.pi])
    best = torch.full_like(dz, far)
    step = max(1, (1 << 22) // R)
    for k in range(0, len(bx), step):
        x, y, w = bx[k:k + step, None], by[k:k + step, None], yaw[k:k + step, None]
        z0 = height(x, y)
        c, s = torch.cos(w), torch.sin(w)
        t0, t1 = torch.zeros(1, device=dev), torch.full((1,), 1e9, device=dev)
        for o, d, l, h in ((-(c * x + s * y), c * dx + s * dy, -half[0, k:k + step, None], half[0, k:k + step, None]),
                           (s * x - c * y, c * dy - s * dx, -half[1, k:k + step, None], half[1, k:k + step, None]),
                           (torch.zeros_like(z0), dz, z0, z0 + tall[k:k + step, None])):
            inv = 1.0 / torch.where(d.abs() < 1e-7, torch.full_like(d, 1e-7), d)
            a, e = (l - o) * inv, (h - o) * inv
            t0, t1 = torch.maximum(t0, torch.minimum(a, e)), torch.minimum(t1, torch.maximum(a, e))
        hit = torch.where((t0 <= t1) & (t0 > 0), t0, torch.full_like(t0, 1e9))
        best = torch.minimum(best, hit.min(0, keepdim=True).values)
    for k in range(nb, nb + nc, step):
        x, y = cx[k:k + step, None], cy[k:k + step, None]
        z0 = height(x, y)
        a, b = dx * dx + dy * dy, dx * x + dy * y
        disc = b * b - a * (x * x + y * y - 0.15 * 0.15)
        t = (b - torch.sqrt(torch.clamp(disc, min=0.0))) / a
        ok = (disc >= 0) & (t > 0) & (t * dz >= z0) & (t * dz <= z0 + 4.0)
        best = torch.minimum(best, torch.where(ok, t, torch.full_like(t, 1e9)).min(0, keepdim=True).values)
    on_ground = t_ground < best
    t = torch.minimum(best, t_ground)
    order = torch.where(t < far, torch.rand(1, R, generator=g, device=dev), torch.full_like(t, 2.0))[0].argsort()
    kept = order[:_kept_points(rings, bins, rate)].sort().values  # where the sky took more: returns at the far end
    n = torch.randn(2, R, generator=g, device=dev) * 0.02
    t = torch.clamp(t, max=far) + n[0]
    z = t * dz + torch.where(on_ground, n[1:], torch.zeros_like(dz))
    p = torch.cat([t * dx, t * dy, z, torch.rand(1, R, generator=g, device=dev)]).T[kept]
    ring = torch.arange(rings - 1, -1, -1, device=dev)[:, None].expand(rings, bins).reshape(R)[kept]
    cfg = lp.SegmenterConfig.default(image_height=rings, image_width=bins, elevation_up_deg=up, elevation_down_deg=down)
    return p.contiguous().cpu().numpy(), ring.cpu().numpy().astype(np.uint16), cfg


def _mixed(seed, k):
    """The k-th scan of an uneven batch: its shape goes round the nine and its return rate over the
    range, the rest comes from the seed."""
    r = np.random.default_rng([seed, k])
    rings, bins, rate = _mixed_shape(k)
    return _scan(int(r.integers(1 << 31)), rings, bins, rate, int(r.integers(10, 201)), int(r.integers(3)),
                 int(r.integers(2)))


def _mixed_shape(k):
    rings, bins = SHAPES[(4 * k + 4) % 9]
    return rings, bins, 0.3 + 0.7 * ((k * 0.618034 + 0.5) % 1.0)


def _cloud(seed, points):
    """An unorganised cloud of exactly `points` points, shuffled: returns of a 128-ring sensor, 5 %
    clutter within 15 m, its density falling with the distance."""
    bins = min(16384, max(512, points // 48))
    a, _, _ = _scan(seed, 128, bins, 1.0, 120, 2, 0)
    r = np.random.default_rng(seed)
    m = points // 20
    rad, c, ang = 15.0 * np.sqrt(r.random(m)), r.uniform(-1, 1, m), r.uniform(0, 2 * np.pi, m)
    s = np.sqrt(1 - c * c)
    clutter = np.stack([rad * s * np.cos(ang), rad * s * np.sin(ang), rad * c, r.random(m)], 1).astype(np.float32)
    a = np.concatenate([a[r.permutation(len(a))[:points - m]], clutter])
    while len(a) < points:  # a few returns more where the sky took too many
        more = a[r.integers(0, len(a), points - len(a))].copy()
        more[:, :3] += r.normal(0, 0.02, (len(more), 3)).astype(np.float32)
        a = np.concatenate([a, more])
    return np.ascontiguousarray(a[r.permutation(points)])


def _obstacles(seed, points):
    """`points` obstacle points in scan order, as the pipeline hands them to the clustering."""
    got, k = [], 0
    while sum(len(a) for a in got) < points:
        a, _, _ = _scan(seed + 7919 * k, 128, 2048, 1.0, 150, 0, 1)
        got.append(a[a[:, 2] > -1.4])
        k += 1
    a = np.concatenate(got)
    keep = np.sort(np.random.default_rng(seed).permutation(len(a))[:points])
    return np.ascontiguousarray(a[keep])


def _footprint(r, n):
    """The points a sensor sees of a parked car or a wall: two sides of a rectangle and some of its
    top, binary32 coordinates held as float64."""
    long, wide = r.uniform(0.5, 20.0), r.uniform(0.1, 3.0)
    t, side = r.random(n), r.random(n)
    x = np.where(side < 0.6, t * long, np.where(side < 0.9, 0.0, t * long))
    y = np.where(side < 0.6, 0.0, np.where(side < 0.9, t * wide, r.random(n) * wide))
    x, y = x + r.normal(0, 0.02, n), y + r.normal(0, 0.02, n)
    yaw, d, a = r.uniform(0, 2 * np.pi), r.uniform(5, 60), r.uniform(0, 2 * np.pi)
    p = np.stack([np.cos(yaw) * x - np.sin(yaw) * y + d * np.cos(a), np.sin(yaw) * x + np.cos(yaw) * y + d * np.sin(a)], 1)
    return np.ascontiguousarray(p.astype(np.float32).astype(np.float64))


# ------------------------------------------------------------------ what a program keeps
class _Results:
    """One scan's result buffers as slices of arrays that hold all scans' results."""

    def __init__(self, all_, at, n, clusters, j, cap, hull_at, hull_cap):
        self.seg = all_["seg"][at:at + n]
        cl = slice(j * cap, (j + 1) * cap)
        p = lp.ptr
        self.out = lp.ScanOutput(p(all_["noise"][at:at + n]), p(self.seg), p(all_["cluster"][at:at + n]), cap, hull_cap,
                                 p(all_["hull_offsets"][j * (cap + 1):(j + 1) * (cap + 1)]),
                                 p(all_["hull_indices"][hull_at:hull_at + hull_cap]), p(all_["z_min"][cl]),
                                 p(all_["z_max"][cl]), p(all_["calipers"][cl]), p(all_["pca"][cl]), 0, 0, 0, 0)


def _buffers(sizes, pinned):
    """Result arrays for scans of these sizes (zeroed), and every scan's view of them."""
    cap = 4096
    hull = [n // 2 + 64 for n in sizes]
    N, S = sum(sizes), len(sizes)

    def zeros(n, dt):
        a = lp.pinned_empty(n * np.dtype(dt).itemsize, np.uint8).view(dt) if pinned else np.zeros(n, dt)
        a.view(np.uint8)[...] = 0
        return a

    all_ = {"noise": zeros(N, np.uint8), "seg": zeros(N, np.uint32), "cluster": zeros(N, np.int32),
            "hull_offsets": zeros(S * (cap + 1), np.uint32), "hull_indices": zeros(sum(hull), np.int32),
            "z_min": zeros(S * cap, np.float32), "z_max": zeros(S * cap, np.float32), "calipers": zeros(S * cap, BOX),
            "pca": zeros(S * cap, BOX)}
    views, at, h = [], 0, 0
    for j, n in enumerate(sizes):
        views.append(_Results(all_, at, n, cap, j, cap, h, hull[j]))
        at, h = at + n, h + hull[j]
    return all_, views


def _boxes(a):
    return {"corners": a["corners"], "area": a["area"], "angle_rad": a["angle_rad"], "is_valid": a["is_valid"]}


def _results(all_):
    signed = {"seg": np.int32, "hull_offsets": np.int32}
    return {k: _boxes(v) if k in ("calipers", "pca") else v.view(signed.get(k, v.dtype)) for k, v in all_.items()}


def _box_list(boxes, capacity):
    return _boxes(_fit(np.frombuffer(b"".join(map(bytes, boxes)), BOX), capacity))


def _fit(a, capacity):
    """The values at the front of an array of a fixed length, as a caller's own buffers hold them."""
    out = np.zeros(capacity, a.dtype)
    out[:len(a)] = a
    return out


_kept = {}


def _context():
    """The context a program opens once and hands every call to."""
    if "ctx" not in _kept:
        _kept["ctx"] = lp.Context(0)
    return _kept["ctx"]


def _server():
    """The serving loop a program starts once."""
    if "server" not in _kept:
        _kept["server"] = lp.Server(0, lp.PipelineConfig.default(), memory_budget_bytes=8 << 30, max_batch_scans=16, slots=3)
    return _kept["server"]


def prepare(case, seed):
    kind, s = case["kind"], {"case": case, "kind": case["kind"]}
    if kind in ("scan", "batch", "prepared", "serve", "filtered"):
        pipe = lp.PipelineConfig.default()
        if kind == "scan":
            scans = [_scan(seed, case["rings"], case["bins"], case["rate"], case["obstacles"], seed % 3, 1)]
        elif kind == "filtered":
            cfg = lp.SegmenterConfig.default(image_height=128, image_width=16384, elevation_up_deg=15.0,
                                             elevation_down_deg=-25.0, assume_unorganized_cloud=1)
            scans = [(_cloud(seed * 64 + k, case["points"]), None, cfg) for k in range(case["scans"])]
            pipe.enable_noise_removal, pipe.noise = 1, lp.NoiseRemoverConfig(3 * 0.17 * math.pi / 180.0, 0.1, 3)
        else:
            scans = [_mixed(seed, k) for k in range(case["scans"])]
        xs, rings, cfgs = [a[0] for a in scans], [a[1] for a in scans], [a[2] for a in scans]
        if case.get("ring") == "computed":
            rings, pipe.compute_ring = None, 1
        elif case.get("ring") == "none" or kind == "filtered":
            rings = None
        if kind == "serve":
            s.update(server=_server(), scans=list(zip(xs, rings, cfgs)))
        elif kind == "prepared":
            s["batch"] = lp.PreparedBatch(_context(), xs, pipe, cfgs, rings)
            s["batch"].capture_graph()
        else:
            pinned = case.get("pinned", True)
            if pinned:
                xs = [lp.pinned_copy(x) for x in xs]
                rings = None if rings is None else [lp.pinned_copy(r) for r in rings]
            s["all"], views = _buffers([len(x) for x in xs], pinned)
            s.update(ctx=_context(), call=lp.BatchCall(xs, pipe, cfgs, rings, outputs=views))
    elif kind == "segment":
        x, _, cfg = _scan(seed, case["rings"], case["bins"], case["rate"], case["obstacles"], seed % 3, 1)
        s.update(x=x, stage=lp.Segmenter(_context(), cfg))
    elif kind == "noise":
        x = _cloud(seed, case["points"])
        cfg = lp.NoiseRemoverConfig.default() if case["default"] else lp.NoiseRemoverConfig(3 * 0.17 * math.pi / 180.0, 0.1, 3)
        s.update(x=np.ascontiguousarray(x[:, :case["stride"]]), stage=lp.NoiseRemover(_context(), cfg))
    elif kind == "cluster":
        x = _obstacles(seed, case["points"])
        cfg = lp.ClustererConfig.default(voxel_grid_elevation_resolution_deg=case["elevation"])
        s.update(x=np.ascontiguousarray(x[:, :case["stride"]]), stage=lp.Clusterer(_context(), cfg))
    elif kind == "polygons":
        s.update(clouds=_polygons(case, seed), stage=lp.Polygonizer(_context()))
    return s


def _polygons(case, seed):
    r = np.random.default_rng(seed)
    n = case["polygons"]
    ratio = math.log(case["largest"] / case["smallest"])
    return [_footprint(r, int(round(case["smallest"] * math.exp(ratio * k / (n - 1))))) for k in range(n)]


def _joined(rs):
    """Results of several scans one after the other, in arrays with room for 1024 clusters a scan."""
    cap = 1024 * len(rs)
    return {"seg": np.concatenate([r.seg_labels for r in rs]).view(np.int32),
            "cluster": np.concatenate([r.cluster_labels for r in rs]),
            "hull_offsets": _fit(np.concatenate([r.hull_offsets for r in rs]).view(np.int32), cap),
            "hull_indices": _fit(np.concatenate([r.hull_indices for r in rs]), 32 * cap),
            "z_min": _fit(np.concatenate([r.z_min for r in rs]), cap),
            "z_max": _fit(np.concatenate([r.z_max for r in rs]), cap),
            "calipers": _box_list([x for r in rs for x in r.obb_calipers], cap),
            "pca": _box_list([x for r in rs for x in r.obb_pca], cap)}


def run(state):
    kind = state["kind"]
    if kind in ("scan", "batch", "filtered"):
        state["call"].run(state["ctx"])
        return _results(state["all"])
    if kind == "prepared":
        b = state["batch"]
        b.upload()
        b.execute()
        return _joined(b.download())
    if kind == "serve":
        srv, scans = state["server"], state["scans"]
        for k, (x, ring, cfg) in enumerate(scans):
            srv.submit(x, ring, cfg, k)
        got = {}
        while len(got) < len(scans):
            for d, r in srv.poll(wait_us=2000):
                got[int(d.tag)] = r
        return _joined([got[k] for k in range(len(scans))])
    if kind == "segment":
        labels = state["stage"].segment(state["x"], want_image=state["case"]["image"]).view(np.int32)
        return [labels, state["stage"].image()] if state["case"]["image"] else labels
    if kind == "noise":
        return state["stage"].filter(state["x"])
    if kind == "cluster":
        return state["stage"].cluster(state["x"])
    p = state["stage"]
    hulls, cal, pca = [], [], []
    for a in state["clouds"]:
        h = p.convexHull(a)
        hulls.append(h)
        cal.append(p.boundingBoxRotatingCalipers(a[h]))
        pca.append(p.boundingBoxPrincipalComponentAnalysis(a[h]))
    return {"hulls": _fit(np.concatenate(hulls), sum(len(a) + 1 for a in state["clouds"])), "calipers": _box_list(cal, len(cal)),
            "pca": _box_list(pca, len(pca))}


# ------------------------------------------------------------------ what a pass cannot do without
def _points(case):
    """Points of a pass."""
    if "points" in case:
        return case["points"] * case.get("scans", 1)
    if "rings" in case:
        return _kept_points(case["rings"], case["bins"], case["rate"])
    return sum(_kept_points(*_mixed_shape(k)) for k in range(case["scans"]))


def work(case):
    kind, n = case["kind"], 0
    if kind == "polygons":
        ratio = math.log(case["largest"] / case["smallest"])
        n = sum(case["smallest"] * math.exp(ratio * k / (case["polygons"] - 1)) for k in range(case["polygons"]))
        return {"bytes": int(16 * n + 200 * case["polygons"]), "flops": int(4 * n * math.log2(n))}
    n = _points(case)
    if kind == "noise":
        return {"bytes": (4 * case["stride"] + 1) * n, "flops": 30 * n}
    if kind == "cluster":
        return {"bytes": (4 * case["stride"] + 4) * n, "flops": 60 * n}
    if kind == "segment":
        return {"bytes": 20 * n + (3 * case["rings"] * case["bins"] if case["image"] else 0), "flops": 100 * n}
    ring = 2 if case.get("ring", "given") == "given" and kind != "filtered" else 0
    # per point: xyzi and ring in, noise, segment and cluster labels out; per cluster (about one in
    # 1500 points): hull, z range, two boxes
    return {"bytes": int((16 + ring + 9) * n + 250 * n / 1500), "flops": 200 * n}


# ------------------------------------------------------------------ the same results in 64 bits
def _hull(a):
    """Monotone chain: counter-clockwise from the lowest (x, y), in binary64."""
    order = np.lexsort((a[:, 1], a[:, 0]))
    pts = [(float(x), float(y)) for x, y in a[order]]

    def half(seq):
        out = []
        for q in seq:
            while len(out) > 1 and ((out[-1][0] - out[-2][0]) * (q[1] - out[-2][1])
                                    - (out[-1][1] - out[-2][1]) * (q[0] - out[-2][0])) <= 0:
                out.pop()
            out.append(q)
        return out

    return np.array(half(pts)[:-1] + half(pts[::-1])[:-1])


def exact(case, seed):
    """Both boxes of each polygon. The other kinds return labels and indices, or are whole pipelines,
    whose ordered vote (one pixel after another) would take minutes here."""
    if case["kind"] != "polygons":
        return None
    areas, corners, pareas = [], [], []
    for a in _polygons(case, seed):
        h = _hull(a)
        c = h - h.mean(0)
        e = np.roll(h, -1, 0) - h
        u = e / np.hypot(e[:, 0], e[:, 1])[:, None]
        along, across = c @ u.T, np.stack([-c[:, 1], c[:, 0]], 1) @ u.T
        areas.append(((along.max(0) - along.min(0)) * (across.max(0) - across.min(0))).min())
        _, v = np.linalg.eigh(c.T @ c / (len(h) - 1))
        m = c @ v
        lo, hi = m.min(0), m.max(0)
        pareas.append((hi - lo).prod())
    return {"hulls": None, "calipers": {"corners": None, "area": np.array(areas), "angle_rad": None, "is_valid": None},
            "pca": {"corners": None, "area": np.array(pareas), "angle_rad": None, "is_valid": None}}
