"""What a user of this framework has it do, as cases whose time can be measured.

Every case goes through the public Python API or the C ABI behind it, on seeded
synthetic clouds: airborne LiDAR over rolling terrain with vegetation, at
UTM-like coordinates.  Results land in arrays that the program owns, sized by
the parameters and filled with -1 beforehand.  A case is a dict of plain
values; ``kind`` names the entry points it calls:

    run     owm_run on a device cloud: the whole path, one call
    host    Context.run_host: points in pinned host memory, seeds out
    stream  Context.run_host_submit / run_host_wait: a stream of clouds
    stages  Context.tree, stage1, stage2, stage3, one call each
    batch   owm_batch_run on tiles that lie back to back in device memory
    serve   Server.submit / wait: tiles of mixed sizes from pinned host memory
    ingest  Context.cloud_parse_xyz on .xyz text, then owm_run

Sizes, window widths, overlaps and cell sizes are those of the repository's
workload configurations, its benchmark and its tests.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import fastowm_gb300 as F

# ---- the cases ----------------------------------------------------------------


def listed():
    return [
        # one small tile: latency and the number of launches count
        {"name": "tile_10k", "kind": "run", "n": 10_007, "density": 20.0, "w": 10, "overlap": 0.8, "b": 20, "leaf": 32,
         "order": "shuffled", "quantum": 0.0, "strips": False},
        # an ordinary plot: 200 m x 250 m at 20 points per square metre
        {"name": "plot_1m", "kind": "run", "n": 1_000_000, "density": 20.0, "w": 10, "overlap": 0.8, "b": 20, "leaf": 32,
         "order": "shuffled", "quantum": 0.0, "strips": False},
        # uneven density, empty holes, heights in whole centimetres (ties), half overlap, odd cell width
        {"name": "strips_20m", "kind": "run", "n": 20_000_000, "density": 31.0, "w": 10, "overlap": 0.5, "b": 15, "leaf": 64,
         "order": "shuffled", "quantum": 0.0, "strips": True},
        # a survey file as delivered: points in flight-line order, coordinates in whole centimetres
        {"name": "scan_40m", "kind": "run", "n": 40_706_503, "density": 12.0, "w": 10, "overlap": 0.8, "b": 20, "leaf": 32,
         "order": "scan", "quantum": 0.01, "strips": False},
        # the largest cloud: 2 km x 2 km at 25 points per square metre
        {"name": "cloud_100m", "kind": "run", "n": 100_000_000, "density": 25.0, "w": 12, "overlap": 0.8, "b": 20, "leaf": 256,
         "order": "shuffled", "quantum": 0.0, "strips": False},
        # a program that holds its points in host memory and makes one call
        {"name": "host_20m", "kind": "host", "n": 20_380_212, "density": 15.0, "w": 10, "overlap": 0.8, "b": 20, "leaf": 32,
         "order": "scan", "quantum": 0.01, "strips": False},
        # the same for a stream of clouds, two runs in flight
        {"name": "stream_4m", "kind": "stream", "n": 4_000_000, "clouds": 4, "density": 25.0, "w": 10, "overlap": 0.8, "b": 20,
         "leaf": 64, "order": "shuffled", "quantum": 0.0, "strips": False},
        # the reference application's functions one by one: index, window minima, seeds, empty cells
        {"name": "stages_2770k", "kind": "stages", "n": 2_770_000, "density": 10.0, "w": 10, "overlap": 0.8, "b": 20, "leaf": 32,
         "radius": 0.0, "order": "shuffled", "quantum": 0.0, "strips": False},
        # the same with the minimum-radius index, on a smaller cloud with small cells
        {"name": "stages_radius_500k", "kind": "stages", "n": 500_009, "density": 20.0, "w": 9, "overlap": 0.5, "b": 6, "leaf": 32,
         "radius": 0.5, "order": "shuffled", "quantum": 0.01, "strips": False},
        # many uneven tiles at once, resident on the device, shapes that come back (graphs on)
        {"name": "batch_128", "kind": "batch", "tiles": 128, "lo": 50_000, "hi": 2_000_000, "density": 0.0, "overlap": 0.8, "b": 20,
         "leaf": 64, "pick": 4},
        # a server's burst: tiles from 10 thousand to 5 million points
        {"name": "serve_48", "kind": "serve", "tiles": 48, "lo": 10_000, "hi": 5_000_000, "density": 0.0, "overlap": 0.8, "b": 20,
         "leaf": 64, "pick": 5},
        # from the text of an .xyz file to its seeds
        {"name": "ingest_4m", "kind": "ingest", "n": 4_000_000, "density": 15.0, "w": 10, "overlap": 0.8, "b": 20, "leaf": 32,
         "order": "scan", "quantum": 0.001, "strips": False},
    ]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "host", "stream", "stages", "batch", "serve", "ingest"])
    c = {"kind": kind, "overlap": rng.choice([0.5, 0.6, 0.8]), "b": rng.choice([0, 6, 15, 20, 25]),
         "leaf": rng.choice([16, 32, 64, 100, 256])}
    if kind in ("batch", "serve"):
        c.update(tiles=rng.randint(2, 128 if kind == "batch" else 48), lo=10_000 if kind == "serve" else 50_000,
                 hi=_log(rng, 200_000, 2_000_000), density=0.0, pick=rng.randint(1, 1 << 20))
        return c
    most = {"run": 80_000_000, "host": 20_000_000, "stream": 4_000_000, "stages": 5_000_000, "ingest": 4_000_000}[kind]
    c.update(n=_log(rng, 10_000, most), density=round(math.exp(rng.uniform(math.log(3.0), math.log(60.0))), 2),
             w=rng.randint(8, 16), order=rng.choice(["shuffled", "scan"]), quantum=rng.choice([0.0, 0.001, 0.01]),
             strips=rng.random() < 0.25)
    if kind == "ingest":
        c["quantum"] = 0.001
    if kind == "stream":
        c["clouds"] = rng.randint(2, 4)
    if kind == "stages":
        c["radius"] = rng.choice([0.0, 0.0, 0.5])
    return c


# ---- inputs --------------------------------------------------------------------

X0, Y0 = 500_000.0, 4_700_000.0  # UTM-like offsets: FP64 is needed to hold a centimetre there


def _side(n, density):
    """Side of the square that holds n points at this density, in whole centimetres."""
    return math.ceil(math.sqrt(n / density) * 100.0) / 100.0


def _points(n, side, seed, x0=X0, y0=Y0, order="shuffled", quantum=0.0, strips=False):
    """n points over a square, [n, 3] float64 on the GPU: terrain of six octaves,
    5 cm of noise, a quarter of the points lifted off the ground by vegetation
    and buildings.  strips: density drawn per 60 m strip, round holes, heights
    in whole centimetres.  scan: flight lines 60 m wide, scan lines across
    them.  quantum: x and y in whole multiples of it."""
    g = torch.Generator(device="cuda").manual_seed(seed)

    def rand(m=n, dtype=torch.float64):
        return torch.rand(m, generator=g, device="cuda", dtype=dtype)

    x, y = rand() * side, rand() * side
    if strips:
        k = max(1, int(math.ceil(side / 60.0)))
        cum = torch.cumsum(5.0 + 55.0 * rand(k), 0)
        i = torch.searchsorted(cum, rand() * cum[-1]).clamp_(max=k - 1)
        x = (i + rand()) * (side / k)
        hx, hy, hr = rand(8) * side, rand(8) * side, (0.04 + 0.11 * rand(8)) * side
        for h in range(8):  # what falls into a hole is drawn again, once
            again = (x - hx[h]) ** 2 + (y - hy[h]) ** 2 < hr[h] ** 2
            y = torch.where(again, (y + 2.0 * hr[h] + rand() * hr[h]) % side, y)
    if order == "scan":
        key = (x / 60.0).floor().mul_(1e6).add_((y / 0.5).floor_())
        idx = torch.argsort(key * 64.0 + (x % 60.0))
        x, y = x[idx], y[idx]
    fx, fy = x.float(), y.float()
    z, a, f = torch.full_like(fx, 100.0), 7.5, 2.0 * math.pi / 160.0
    for p in (rand(12, torch.float32) * (2.0 * math.pi)).view(6, 2).tolist():
        z += a * torch.sin(fx * f + p[0]) * torch.cos(fy * f + p[1])
        a, f = a * 0.5, f * 2.0
    z = z.double() + 0.05 * torch.randn(n, generator=g, device="cuda", dtype=torch.float32).double()
    lift = rand(dtype=torch.float32)
    z += torch.where(lift < 0.25, lift * 98.0 + 0.5, torch.zeros_like(lift)).double()
    if strips:
        z = torch.round(z * 100.0) / 100.0
    x, y = x + x0, y + y0
    if quantum:
        m = round(1.0 / quantum)
        x, y = torch.round(x * m) / m, torch.round(y * m) / m
    return torch.stack([x, y, z], 1)


def _box(side, x0=X0, y0=Y0):
    """The cloud's box as its file header states it: the surveyed square."""
    return F.Bbox(x0, y0, x0 + side, y0 + side)


def _pinned(t):
    """The same points in pinned host memory, as the numpy array that the API takes."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _cfg(c, w=None):
    radius = c.get("radius", 0.0)
    return F.run_cfg(c["w"] if w is None else w, c["overlap"], c["b"], c["leaf"],
                     F.OWM_TREE_MIN_RADIUS if radius else F.OWM_TREE_MAX_NUMBER, radius or 0.1)


def _ids(n):
    """A result array of n ids, none yet."""
    return np.full(n, -1, dtype=np.int64)


def _room(box, n, cfg):
    p = F.params(box, n, cfg.wsize, cfg.overlap, cfg.bsize)
    return p.ncells + p.ngrid + 1


def _tile_shapes(c):
    """(points, side, Wsize) of every tile: counts log-uniform, squares of 100 to 500 m."""
    r = np.random.default_rng(c["pick"])
    n = np.exp(r.uniform(math.log(c["lo"]), math.log(c["hi"]), c["tiles"])).astype(np.int64)
    return list(zip(n.tolist(), np.floor(r.uniform(100, 500, c["tiles"])).tolist(), r.integers(8, 17, c["tiles"]).tolist()))


def _text(t, box):
    """.xyz text of the points: five header lines, then fixed-width %.3f lines."""
    n = t.shape[0]
    head = "%d\n%.3f\n%.3f\n%.3f\n%.3f\n" % (n, box.min_x, box.max_x, box.min_y, box.max_y)
    cols = []
    for k, width in ((0, 6), (1, 7), (2, 4)):  # digits before the point
        v = torch.round(t[:, k] * 1000.0).long()
        digits = [(v // 10 ** p) % 10 + 48 for p in range(width + 2, -1, -1)]
        digits.insert(width, torch.full_like(v, 46))
        cols += digits + [torch.full_like(v, 10 if k == 2 else 32)]
    body = torch.stack([q.to(torch.uint8) for q in cols], 1).reshape(-1)
    out = torch.empty(len(head) + body.numel(), dtype=torch.uint8, pin_memory=True)
    out[:len(head)] = torch.from_numpy(np.frombuffer(head.encode(), np.uint8).copy())
    out[len(head):].copy_(body)
    return out.numpy()


_shared = {}


def _context():
    """One context for the program, as a program keeps one."""
    if "ctx" not in _shared:
        _shared["ctx"] = F.Context(0)
    return _shared["ctx"]


def prepare(case, seed):
    c, ctx = case, _context()
    s = {"case": c, "ctx": ctx, "kind": c["kind"]}
    if "n" in c:
        n, side = c["n"], _side(c["n"], c["density"])
        how = dict(order=c["order"], quantum=c["quantum"], strips=c["strips"])
        box, cfg = _box(side), _cfg(c)
        s.update(box=box, cfg=cfg, seeds=_ids(_room(box, n, cfg)))
    if c["kind"] in ("run", "stages"):
        t = _points(n, side, seed, **how)
        h = C.c_void_p()
        torch.cuda.synchronize()
        rc = F.lib().owm_cloud_create(ctx.handle, C.cast(t.data_ptr(), C.POINTER(C.c_double)), n, C.byref(box), C.byref(h))
        if rc:
            raise F.OwmError(rc, "cloud_create")
        s["cloud"] = F.Cloud(ctx, h, n, box)
        if c["kind"] == "stages":
            p = F.params(box, n, c["w"], c["overlap"], c["b"])
            s.update(params=p, llp=_ids(p.ncells), stage3=_ids(p.ngrid))
    elif c["kind"] == "host":
        s["xyz"] = _pinned(_points(n, side, seed, **how))
    elif c["kind"] == "stream":
        s["clouds"] = [(_pinned(_points(n, side, seed * 64 + k, **how)), box, cfg, _ids(s["seeds"].size)) for k in range(c["clouds"])]
    elif c["kind"] == "ingest":
        t = _points(n, side, seed, **how)
        t[:, 2] = torch.round(t[:, 2] * 1000.0) / 1000.0
        s["text"] = _text(t, box)
    else:
        tiles = []
        for k, (n, side, w) in enumerate(_tile_shapes(c)):
            x0, y0 = 400_000.0 + (k % 64) * 1000.0, 4_400_000.0 + (k // 64) * 1000.0
            box, cfg = _box(side, x0, y0), _cfg(c, w)
            tiles.append((_points(n, side, seed * 4096 + k, x0, y0), box, cfg, _room(box, n, cfg)))
        if c["kind"] == "serve":
            s["server"] = F.Server(0, copy_on_submit=False)
            s["tiles"] = [(_pinned(t), box, cfg, _ids(room)) for t, box, cfg, room in tiles]
        else:
            s["points"] = torch.cat([t for t, _, _, _ in tiles])
            s["tiles"], at = (F.TileDesc * len(tiles))(), 0
            for k, (t, box, cfg, _) in enumerate(tiles):
                here = C.cast(s["points"].data_ptr() + 24 * at, C.POINTER(C.c_double))
                s["tiles"][k] = F.TileDesc(here, t.shape[0], box, cfg)
                at += t.shape[0]
            s.update(batch=F.Batch(ctx), seeds=_ids(sum(room for _, _, _, room in tiles)), offsets=_ids(len(tiles) + 1))
            s["batch"].set_graphs(True)
    torch.cuda.synchronize()
    return s


# ---- one pass ------------------------------------------------------------------

_i64 = C.POINTER(C.c_int64)


def _whole_path(ctx, cloud, cfg, seeds):
    n, info = C.c_int64(), F.RunInfo()
    rc = F.lib().owm_run(ctx.handle, cloud.handle, C.byref(cfg), seeds.ctypes.data_as(_i64), seeds.size, C.byref(n), C.byref(info))
    if rc:
        raise F.OwmError(rc, "run")
    return {"seeds": seeds, "count": n.value}


def run(state):
    s, ctx = state, state["ctx"]
    if s["kind"] == "run":
        return _whole_path(ctx, s["cloud"], s["cfg"], s["seeds"])
    if s["kind"] == "ingest":
        cloud = ctx.cloud_parse_xyz(s["text"])
        got = _whole_path(ctx, cloud, s["cfg"], s["seeds"])
        cloud.close()
        return got
    if s["kind"] == "host":
        got = ctx.run_host(s["xyz"], s["box"], s["cfg"], out=s["seeds"])
        return {"seeds": s["seeds"], "count": got.size}
    if s["kind"] == "stream":
        counts, flying = [], []
        for cloud in s["clouds"]:
            flying.append(ctx.run_host_submit(*cloud))
            if len(flying) == 2:
                counts.append(ctx.run_host_wait(flying.pop(0)).size)
        counts += [ctx.run_host_wait(t).size for t in flying]
        return {"seeds": [c[3] for c in s["clouds"]], "count": counts}
    if s["kind"] == "stages":
        t, p = s["cfg"].tree, s["params"]
        tree = ctx.tree(s["cloud"], t.policy, t.max_number, t.min_radius)
        win = ctx.stage1(tree, p)
        llp = ctx.stage2(win.copy(), p.overlap)  # the call sorts its argument in place
        s3 = ctx.stage3(tree, p, llp)
        info = tree.info()
        tree.close()
        s["llp"][:llp.size] = llp
        s["stage3"][:s3.size] = s3
        return {"windows": win, "llp": s["llp"], "stage3": s["stage3"], "points": info.root_count, "lowest": info.root_min_id}
    if s["kind"] == "serve":
        tickets = [s["server"].submit(xyz, box, cfg) for xyz, box, cfg, _ in s["tiles"]]
        for ticket, (_, _, _, ids) in zip(tickets, s["tiles"]):
            got, _ = s["server"].wait(ticket, ids.size)
            ids[:got.size] = got
        return [ids for _, _, _, ids in s["tiles"]]
    rc = F.lib().owm_batch_run(s["batch"].handle, s["tiles"], len(s["tiles"]), s["seeds"].ctypes.data_as(_i64), s["seeds"].size,
                               s["offsets"].ctypes.data_as(_i64), None)
    if rc:
        raise F.OwmError(rc, "batch_run")
    return {"offsets": s["offsets"], "seeds": s["seeds"]}


# ---- what a pass cannot do without ----------------------------------------------


def work(case):
    """Each point's x, y, z read once (or its text), each result written once:
    a seed for about one window in seven (8 bytes), for the stage calls also the
    window minima.  Operations: four comparisons with a box and one of heights
    for each point and each of the two grids."""
    c = case
    if c["kind"] in ("batch", "serve"):
        shapes = _tile_shapes(c)
        n = sum(k for k, _, _ in shapes)
        windows = sum((side / (w * (1.0 - c["overlap"]))) ** 2 for _, side, w in shapes)
        return {"bytes": 24.0 * n + 8.0 * windows / 7.0, "flops": 10.0 * n}
    n = c["n"] * c.get("clouds", 1)
    windows = n / c["density"] / (c["w"] * (1.0 - c["overlap"])) ** 2
    per_point = 37.0 if c["kind"] == "ingest" else 24.0
    out = 8.0 * windows * (1.0 if c["kind"] == "stages" else 0.0) + 8.0 * windows / 7.0
    return {"bytes": per_point * n + out, "flops": 10.0 * n}


def exact(case, seed):
    """Every output is a list of point numbers or a count: whole numbers, which
    have no rounding to be compared with."""
    return None
