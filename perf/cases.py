"""The work that programs have this library do, as cases that can be timed and checked.

Every case is one whole call sequence of a user's program through the Python binding of
the C ABI (gvx.Grid, gvx.Batch, gvx.radix_sort): points in device or host memory in, channels
of the brick atlas (or gradients, or sorted pairs) out.  The kinds:

  frame     RebuildTopology (full) + FinishTopology + UpdateAtlas + InsertPoints + splat +
            UpdateApron, the frame of a simulation or of a live point source
  scatter   the same frame with ScatterDensity and averaged point colours
  surface   a fluid surface: one full and then incremental rebuilds of moving points, subcell
            lists, a gather, apron and smoothing
  fusion    depth-camera frames accumulated into one growing volume
  cloud     a 16-bit point cloud decoded and turned into a smoothed level set
  batch     many point clouds of uneven size in one batched frame
  gradient  one step of fitting points to a density: splat, loss gradient, adjoint
  sort      RadixSortByByte on its own

exact() restates the outputs in 64-bit torch: the active bricks in pool order, the voxel sums,
the apron copies.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "gvdb-voxels_gb300"))

import gvx  # noqa: E402

LEVELS = (3, 3, 3, 3, 5)  # 8^3 bricks, the configuration of the samples and of the benchmark


def listed():
    return [
        # a live source of few points (a tracked object, a small emitter): launches and waits
        {"name": "live_6k", "kind": "frame", "n": 6_000, "box": "56x48x64", "jitter": 0.0, "mode": "trilinear",
         "radius": 1.0, "vel": False, "weight": True, "brick": 3, "source": "packed"},
        # the small uniform volume of the plain configuration
        {"name": "plain_100k", "kind": "frame", "n": 100_000, "box": "256x256x256", "jitter": 0.0,
         "mode": "trilinear", "radius": 1.0, "vel": False, "weight": False, "brick": 3, "source": "packed"},
        # the dam-break slab: the headline frame, density and velocity
        {"name": "sph_4m", "kind": "frame", "n": 4_000_000, "box": "512x256x1024", "jitter": 0.3, "mode": "cubic",
         "radius": 2.0, "vel": True, "weight": False, "brick": 3, "source": "packed"},
        # a simulation that keeps its particles on the host: upload, frame, brick table read back
        {"name": "sph_host_777k", "kind": "frame", "n": 777_777, "box": "300x150x400", "jitter": 0.3, "mode": "cubic",
         "radius": 2.0, "vel": True, "weight": True, "brick": 3, "source": "host"},
        # interleaved particle records into 16^3 bricks, a wide density kernel
        {"name": "records_16_300k", "kind": "frame", "n": 300_001, "box": "333x127x250", "jitter": 0.0, "mode": "cubic",
         "radius": 3.5, "vel": False, "weight": False, "brick": 4, "source": "records"},
        # ScatterDensity with averaged colours, as the sample does it
        {"name": "scatter_1m", "kind": "scatter", "n": 1_000_003, "box": "320x256x320", "radius": 2.0, "avg": True},
        # a fluid surface over three steps: the default (incremental) rebuild, gathers, smoothing
        {"name": "surface_400k", "kind": "surface", "n": 400_000, "box": "180x60x180", "steps": 3, "subcell": 4,
         "radius": 1.0, "op": "levelset"},
        # five frames of a 640x480 depth camera into a growing 2048^3 volume
        {"name": "fusion_5x640x480", "kind": "fusion", "frames": 5, "width": 640, "height": 480},
        # a scanned cloud of 16-bit points to a smoothed level set
        {"name": "cloud_6m", "kind": "cloud", "n": 6_000_000, "extent": 1024.0},
        # clouds of uneven size, all in one frame
        {"name": "batch_24", "kind": "batch", "clouds": 24, "nmin": 10_000, "nmax": 1_000_000, "cloud_seed": 7},
        # fitting a million points of differing radii to a density
        {"name": "gradient_1m", "kind": "gradient", "n": 1_000_000, "box": "496x496x496", "rmin": 1.0, "rmax": 3.0},
        # sorting key/value pairs that a program made itself
        {"name": "sort_3m", "kind": "sort", "n": 3_000_001, "bits": 30},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, n, lo, hi, most=1100):
    """a box of about n / density voxels, its sides unequal, density log-uniform in [lo, hi]"""
    vol = n / math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a, b = rng.uniform(0.6, 1.6), rng.uniform(0.6, 1.6)
    s = vol ** (1.0 / 3.0)
    return "%dx%dx%d" % tuple(max(24, min(most, int(s * f))) for f in (a, b, 1.0 / (a * b)))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "scatter", "surface", "fusion", "cloud", "batch", "gradient",
                       "sort"])
    if kind == "frame":
        n = _log(rng, 3_000, 2_500_000)
        cubic = rng.random() < 0.6
        return {"kind": kind, "n": n, "box": _box(rng, n, 0.02, 0.2), "jitter": rng.choice([0.0, 0.3]),
                "mode": "cubic" if cubic else "trilinear",
                "radius": rng.choice([1.5, 2.0, 2.0, 3.0]) if cubic else 1.0, "vel": rng.random() < 0.5,
                "weight": rng.random() < 0.5, "brick": rng.choice([3, 3, 3, 4]),
                "source": rng.choice(["packed", "packed", "records", "host"])}
    if kind == "scatter":
        n = _log(rng, 5_000, 1_500_000)
        return {"kind": kind, "n": n, "box": _box(rng, n, 0.02, 0.2), "radius": rng.choice([1.5, 2.0, 3.0]),
                "avg": rng.random() < 0.5}
    if kind == "surface":
        n = _log(rng, 5_000, 500_000)
        return {"kind": kind, "n": n, "box": _box(rng, n, 0.1, 0.4, 400), "steps": rng.randint(2, 4),
                "subcell": rng.choice([4, 4, 2]), "radius": 1.0, "op": rng.choice(["levelset", "density"])}
    if kind == "fusion":
        w = _log(rng, 160, 640)
        return {"kind": kind, "frames": rng.randint(3, 6), "width": w, "height": w * 3 // 4}
    if kind == "cloud":
        return {"kind": kind, "n": _log(rng, 50_000, 4_000_000), "extent": float(rng.choice([512, 768, 1024]))}
    if kind == "batch":
        return {"kind": kind, "clouds": rng.randint(3, 24), "nmin": _log(rng, 2_000, 10_000),
                "nmax": _log(rng, 50_000, 600_000), "cloud_seed": rng.randrange(1 << 20)}
    if kind == "gradient":
        n = _log(rng, 10_000, 900_000)
        return {"kind": kind, "n": n, "box": _box(rng, n, 0.005, 0.05, 496), "rmin": 1.0,
                "rmax": round(rng.uniform(1.5, 3.0), 2)}
    return {"kind": kind, "n": _log(rng, 2_000, 3_000_000), "bits": rng.randint(12, 32)}


# --------------------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFF)
    return g


def _box_of(case):
    return [float(v) for v in case["box"].split("x")]


def _rand(n, k, g):
    return torch.rand((n, k), generator=g, device="cuda", dtype=torch.float32)


def _randn(n, k, g):
    return torch.randn((n, k), generator=g, device="cuda", dtype=torch.float32)


def _uniform(case, g):
    """positions of a filled box, as a fluid or a volume of samples has them"""
    pos = _rand(case["n"], 3, g) * torch.tensor(_box_of(case), device="cuda")
    if case.get("jitter"):
        pos = pos + case["jitter"] * _randn(case["n"], 3, g)
    return pos.contiguous()


def _surface_points(n, extent, g):
    """points scanned from spheres and a floor (the same scene every time), with noise"""
    c = 0.5 * extent
    scene = _gen(5)
    centre = c + (_rand(8, 3, scene) - 0.5) * (0.5 * extent)
    rad = (0.03 + 0.09 * _rand(8, 1, scene)) * extent
    which = torch.randint(0, 10, (n,), generator=g, device="cuda")
    d = _randn(n, 3, g)
    d = d / d.norm(dim=1, keepdim=True).clamp_min(1e-6)
    ball = centre[which.clamp_max(7)] + d * rad[which.clamp_max(7)]
    floor = torch.stack([_rand(n, 1, g)[:, 0] * extent, torch.full((n,), 0.2 * extent, device="cuda"),
                         _rand(n, 1, g)[:, 0] * extent], 1)
    p = torch.where((which >= 8)[:, None], floor, ball) + 0.5 * _randn(n, 3, g)
    return p.clamp(2.0, extent - 3.0)


def _depth_frames(case, seed):
    """(positions, confidence) of each frame of a pinhole camera on a circle around spheres above a floor;
    the scene is the same every time, the camera's start and the noise are the seed's"""
    g, scene = _gen(seed), _gen(3)
    start = 0.01 * float(_rand(1, 1, g))
    w, h = case["width"], case["height"]
    ext = 2048.0
    c0 = torch.full((3,), 0.5 * ext, device="cuda")
    sc = c0 + (_rand(8, 3, scene) - 0.5) * 600.0
    sr = 60.0 + 120.0 * _rand(8, 1, scene)[:, 0]
    f = 525.0 * w / 640.0
    v, u = torch.meshgrid(torch.arange(h, device="cuda", dtype=torch.float32),
                          torch.arange(w, device="cuda", dtype=torch.float32), indexing="ij")
    dc = torch.stack([(u - 0.5 * w) / f, (v - 0.5 * h) / f, torch.ones_like(u)], -1).reshape(-1, 3)
    dc = dc / dc.norm(dim=1, keepdim=True)
    out = []
    for k in range(case["frames"]):
        ang = start + 2.0 * math.pi * k / 30.0
        cam = c0 + torch.tensor([700.0 * math.cos(ang), 150.0, 700.0 * math.sin(ang)], device="cuda")
        fwd = (c0 - cam) / (c0 - cam).norm()
        right = torch.linalg.cross(fwd, torch.tensor([0.0, 1.0, 0.0], device="cuda"))
        right = right / right.norm()
        up = torch.linalg.cross(right, fwd)
        d = dc[:, :1] * right - dc[:, 1:2] * up + dc[:, 2:3] * fwd
        t = torch.full((len(d),), math.inf, device="cuda")
        nrm = torch.zeros_like(d)
        for s in range(8):
            oc = cam - sc[s]
            b = d @ oc
            disc = b * b - (oc @ oc - sr[s] * sr[s])
            th = torch.where(disc > 0, -b - disc.clamp_min(0).sqrt(), math.inf)
            hit = (th > 1.0) & (th < t)
            t = torch.where(hit, th, t)
            nrm = torch.where(hit[:, None], (cam + torch.where(hit, th, 0.0)[:, None] * d - sc[s]) / sr[s], nrm)
        th = (c0[1] - 350.0 - cam[1]) / d[:, 1]
        hit = (d[:, 1].abs() > 1e-6) & (th > 1.0) & (th < t)
        t = torch.where(hit, th, t)
        nrm = torch.where(hit[:, None], torch.tensor([0.0, 1.0, 0.0], device="cuda"), nrm)
        ok = t < 2000.0
        p = cam + t[ok, None] * d[ok] + 0.5 * _randn(int(ok.sum()), 3, g)
        conf = (nrm[ok] * d[ok]).sum(1).abs()
        keep = ((p >= 0) & (p < ext)).all(1)
        out.append((p[keep].contiguous(), conf[keep].contiguous()))
    return out


def _cloud_sizes(case):
    rng = np.random.default_rng(case["cloud_seed"])
    return [int(v) for v in np.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"]), case["clouds"]))]


def _clouds(case, seed):
    """(positions, weights) of every cloud: Gaussian blobs, their places and widths the case's, the points the seed's"""
    g, shape = _gen(seed), _gen(case["cloud_seed"])
    return [_blobs(n, g, shape) for n in _cloud_sizes(case)]


def _blobs(n, g, shape):
    k = int(torch.randint(1, 17, (1,), generator=shape, device="cuda"))
    centre = 128.0 + 768.0 * _rand(k, 3, shape)
    sig = 4.0 + 60.0 * _rand(k, 1, shape)
    comp = torch.randint(0, k, (n,), generator=g, device="cuda")
    return (centre[comp] + _randn(n, 3, g) * sig[comp]).clamp(0.0, 1023.999).contiguous(), 0.5 + _rand(n, 1, g)[:, 0]


def _inputs(case, seed):
    """every input tensor of a case (device memory), from the seed alone"""
    g = _gen(seed)
    k = case["kind"]
    if k == "frame":
        return {"pos": _uniform(case, g), "vel": _randn(case["n"], 3, g) if case["vel"] else None,
                "w": (0.5 + _rand(case["n"], 1, g)[:, 0]) if case["weight"] else None}
    if k == "scatter":
        return {"pos": _uniform(case, g),
                "clr": torch.randint(0, 256, (case["n"], 4), generator=g, device="cuda", dtype=torch.uint8)}
    if k == "surface":
        # a body of fluid in a wider tank, carried along and stirred by smooth waves
        p = _uniform(case, g) + 16.0
        phase = 6.0 * _rand(3, 1, g)[:, 0]
        vel = torch.stack([2.0 + torch.sin(p[:, 2] / 17.0 + phase[0]), torch.cos(p[:, 0] / 13.0 + phase[1]),
                           torch.sin(p[:, 0] / 19.0 + phase[2])], 1)
        return {"pos": [(p + 1.5 * s * vel).contiguous() for s in range(case["steps"])],
                "clr": torch.randint(0, 256, (case["n"], 4), generator=g, device="cuda", dtype=torch.uint8)}
    if k == "cloud":
        p = _surface_points(case["n"], case["extent"], g)
        q = (p * (65535.0 / case["extent"])).round().to(torch.int32)
        return {"q": torch.where(q >= 32768, q - 65536, q).to(torch.int16).contiguous()}  # the bits of uint16
    if k == "gradient":
        n = case["n"]
        lo = 8.0
        pos = (lo + _rand(n, 3, g) * torch.tensor(_box_of(case), device="cuda")).contiguous()
        w = _rand(n, 1, g)[:, 0].contiguous()
        r = (case["rmin"] + (case["rmax"] - case["rmin"]) * _rand(n, 1, g)[:, 0]).contiguous()
        other = (pos + 0.25 * _randn(n, 3, g)).clamp_min(0.0)
        return {"pos": pos, "w": w, "r": r, "other": other}
    if k == "sort":
        b = case["bits"]
        keys = torch.randint(0, 1 << b, (case["n"],), generator=g, device="cuda", dtype=torch.int64)
        keys = torch.where(keys >= 1 << 31, keys - (1 << 32), keys).to(torch.int32)  # the bits of uint32
        return {"keys": keys, "vals": torch.arange(case["n"], device="cuda", dtype=torch.int32)}
    raise ValueError(k)


class _DeviceView:
    """channel memory for torch; holds the grid, so that the memory lives as long as a tensor of it"""

    def __init__(self, grid, ptr, nbytes):
        self.grid = grid
        self.__cuda_array_interface__ = {"shape": (nbytes // 4,), "typestr": "<f4", "data": (ptr, False),
                                         "version": 2}


def _channel(st, g, chan, dtype=torch.float32):
    """the channel's device memory as a tensor, where it lies (the view made again when it moved or grew)"""
    at = (g.channel_device_ptr(chan), dtype)
    views = st.setdefault("views", {})
    if views.get((id(g), chan), (None, None))[0] != at:
        views[(id(g), chan)] = (at, torch.as_tensor(_DeviceView(g, *at[0]), device="cuda").view(dtype))
    return views[(id(g), chan)][1]


def _grid(levels, channels, layers):
    """a grid whose atlas starts with room for 16 x 16 x layers bricks"""
    g = gvx.Grid(0)
    g.configure(levels)
    g.set_channel_default(16, 16, layers)
    for c, t in channels:
        g.add_channel(c, t, 1)
    return g


def _topo_radius(case):
    return 1.0 if case["mode"] == "trilinear" else float(math.ceil(case["radius"]))


# --------------------------------------------------------------------------- prepare / run

def prepare(case, seed):
    k = case["kind"]
    if k == "fusion":
        g = _grid(LEVELS, [(0, gvx.T_FLOAT), (1, gvx.T_FLOAT)], _layers(case)[0])
        return {"case": case, "grid": g, "frames": _depth_frames(case, seed)}
    if k == "batch":
        clouds, grids = _clouds(case, seed), []
        for (p, w), layers in zip(clouds, _layers(case)):
            g = _grid(LEVELS, [(0, gvx.T_FLOAT)], layers)
            g.set_points(len(p), p)
            g.set_point_attribs(weight=w)
            grids.append(g)
        b = gvx.Batch(0)
        b.set_grids(grids)
        return {"case": case, "batch": b, "grids": grids, "clouds": clouds}
    inp = _inputs(case, seed)
    st = {"case": case, "in": inp}
    layers = _layers(case)[0]
    if k == "frame":
        st["grid"] = _grid((case["brick"],) + LEVELS[1:],
                           [(0, gvx.T_FLOAT)] + ([(1, gvx.T_FLOAT3)] if case["vel"] else []), layers)
        if case["source"] == "records":
            # one record a particle: position, velocity, colour
            rec = torch.zeros((case["n"], 7), device="cuda")
            rec[:, 0:3] = inp["pos"]
            if case["vel"]:
                rec[:, 3:6] = inp["vel"]
            st["rec"] = rec
        elif case["source"] == "host":
            st["host"] = {a: v.cpu().pin_memory().numpy() for a, v in inp.items() if v is not None}
    elif k == "scatter":
        st["grid"] = _grid(LEVELS, [(0, gvx.T_FLOAT), (1, gvx.T_UCHAR4), (3, gvx.T_UCHAR4)], layers)
    elif k == "surface":
        g = _grid(LEVELS, [(0, gvx.T_FLOAT), (1, gvx.T_UCHAR4)], layers)
        # the simulation has been running: its first two builds are full ones
        g.set_points(case["n"], inp["pos"][0])
        g.rebuild_topology(case["n"], case["radius"], mode=gvx.TOPO_FULL)
        g.rebuild_topology(case["n"], case["radius"], mode=gvx.TOPO_AUTO)
        st["grid"] = g
    elif k == "cloud":
        st["grid"] = _grid(LEVELS, [(0, gvx.T_FLOAT)], layers)
        st["pos"] = torch.empty((case["n"], 3), device="cuda")
    elif k == "gradient":
        g = _grid(LEVELS, [(0, gvx.T_FLOAT)], layers)
        g.set_stream(torch.cuda.current_stream().cuda_stream)  # the program's torch operations and the grid in order
        n = case["n"]
        # the bricks of the fitted volume stay the same over the steps; the target is the
        # density of a perturbed copy of the points
        g.set_points(n, inp["pos"])
        g.rebuild_topology(n, 3.0, mode=gvx.TOPO_FULL)
        g.update_atlas()
        bricks = _full_bricks(inp["pos"], 3.0, LEVELS)
        rho = _splat64(inp["other"], inp["w"], inp["r"], "cubic", bricks, 8)
        st["target"] = _padded(rho, bricks, 8, 256 * layers).float().reshape(-1)
        st["grad"] = [torch.empty((n, 3), device="cuda"), torch.empty(n, device="cuda"), torch.empty(n, device="cuda")]
        st["grid"] = g
    elif k == "sort":
        st["grid"] = gvx.Grid(0)
        st["out"] = [torch.empty_like(inp["keys"]), torch.empty_like(inp["vals"])]
    return st


def run(st):
    case = st["case"]
    return _RUN[case["kind"]](case, st)


def _run_frame(case, st):
    g, n, inp = st["grid"], case["n"], st["in"]
    if case["source"] == "host":
        h = st["host"]
        g.commit_points_host(h["pos"], vel=h.get("vel"), weight=h.get("w"))
    elif case["source"] == "records":
        g.set_points(n, st["rec"], 0, 28, vel=st["rec"] if case["vel"] else None, vel_offset=12, vel_stride=28)
        g.set_point_attribs(weight=inp["w"])
    else:
        g.set_points(n, inp["pos"], vel=inp["vel"])
        g.set_point_attribs(weight=inp["w"])
    g.rebuild_topology(n, _topo_radius(case), mode=gvx.TOPO_FULL)
    g.finish_topology()
    g.update_atlas()
    g.insert_points(n)
    g.splat(gvx.SPLAT_TRILINEAR if case["mode"] == "trilinear" else gvx.SPLAT_CUBIC, n, case["radius"],
            chan_density=0, chan_vel=1 if case["vel"] else -1)
    g.update_apron(0, 0.0)
    out = {"density": _channel(st, g, 0)}
    if case["vel"]:
        g.update_apron(1, 0.0)
        out["velocity"] = _channel(st, g, 1)
    if case["source"] == "host":
        out["bricks"] = g.read_atlas_map()
    return out


def _run_scatter(case, st):
    g, n = st["grid"], case["n"]
    g.set_points(n, st["in"]["pos"], clr=st["in"]["clr"])
    g.rebuild_topology(n, case["radius"], mode=gvx.TOPO_FULL)
    g.finish_topology()
    g.update_atlas()
    chan = 1 if case["avg"] else 3
    g.clear_channel(0)
    g.clear_channel(chan)
    g.insert_points(n)
    g.scatter_density(n, case["radius"], expand=True, avg_color=case["avg"])
    g.update_apron(0, 0.0)
    g.update_apron(chan, 0.0)
    return {"density": _channel(st, g, 0), "colour": _channel(st, g, chan, torch.uint8)}


def _run_surface(case, st):
    g, n, r, sc = st["grid"], case["n"], case["radius"], case["subcell"]
    level = case["op"] == "levelset"
    bv = 3.0 if level else 0.0
    for s, pos in enumerate(st["in"]["pos"]):
        g.set_points(n, pos, clr=st["in"]["clr"])
        g.rebuild_topology(n, r, mode=gvx.TOPO_FULL if s == 0 else gvx.TOPO_AUTO)
        g.finish_topology()
        g.update_atlas()
        g.clear_channel(0)
        ln = g.insert_points_subcell(sc, n, r)
        if level:
            g.gather_levelset(sc, n, r, ln, chan=0, chan_clr=1)
        else:
            g.gather_density(sc, n, r, ln, chan=0, chan_clr=1)
        g.update_apron(0, bv)
        g.update_apron(1, 0.0)
        g.compute(gvx.FUNC_SMOOTH, 0, 2, (1.0, 0.0, 0.0), True, True, bv)
    return {"surface": _channel(st, g, 0), "colour": _channel(st, g, 1, torch.uint8)}


def _run_fusion(case, st):
    g = st["grid"]
    g.clear()
    g.clear_channel(0)
    g.clear_channel(1)
    for pos, conf in st["frames"]:
        n = len(pos)
        g.set_points(n, pos)
        g.set_point_attribs()
        g.rebuild_topology(n, 1.0, mode=gvx.TOPO_ACCUMULATE)
        g.update_atlas()
        g.insert_points(n)
        g.splat(gvx.SPLAT_TRILINEAR, n, 1.0, chan_density=0, accum=True)
        g.set_point_attribs(weight=conf)
        g.splat(gvx.SPLAT_TRILINEAR, n, 1.0, chan_density=1, accum=True)
        g.update_apron(0, 0.0)
        g.update_apron(1, 0.0)
    return {"density": _channel(st, g, 0), "confidence": _channel(st, g, 1)}


def _run_cloud(case, st):
    g, n = st["grid"], case["n"]
    d = case["extent"] / 65535.0
    g.convert_and_transform(st["in"]["q"], 2, st["pos"], n, (0.0, 0.0, 0.0), (d, d, d))
    g.set_points(n, st["pos"])
    g.rebuild_topology(n, 2.0, mode=gvx.TOPO_FULL)
    g.finish_topology()
    g.update_atlas()
    ln = g.insert_points_subcell_fp16(4, n, 1.0)
    g.gather_levelset_fp16(4, n, 1.0, ln, chan=0)
    g.update_apron(0, 3.0)
    g.compute(gvx.FUNC_SMOOTH, 0, 1, (1.0, 0.0, 0.0), True, True, 3.0)
    return {"levelset": _channel(st, g, 0)}


def _run_batch(case, st):
    st["batch"].frame(1.0, gvx.SPLAT_TRILINEAR, 1.0, graph=True)
    return [_channel(st, g, 0) for g in st["grids"]]


def _run_gradient(case, st):
    g, n, inp = st["grid"], case["n"], st["in"]
    g.set_points(n, inp["pos"])
    g.set_point_attribs(weight=inp["w"], radius=inp["r"])
    g.splat(gvx.SPLAT_CUBIC, n, 1.0, chan_density=0)
    rho = _channel(st, g, 0)
    dl = torch.sub(rho, st["target"]).mul_(2.0)
    gp, gw, gr = st["grad"]
    g.splat_backward(gvx.SPLAT_CUBIC, n, 1.0, dl, gp, gw, gr)
    return {"density": rho, "dpos": gp, "dweight": gw, "dradius": gr}


def _run_sort(case, st):
    gvx.radix_sort(st["grid"], st["in"]["keys"], st["in"]["vals"], st["out"][0], st["out"][1], case["n"], case["bits"])
    return {"keys": st["out"][0], "vals": st["out"][1]}


_RUN = {"frame": _run_frame, "scatter": _run_scatter, "surface": _run_surface, "fusion": _run_fusion,
        "cloud": _run_cloud, "batch": _run_batch, "gradient": _run_gradient, "sort": _run_sort}


# --------------------------------------------------------------------------- restatement in 64 bits

_BIG = 1 << 21


def _pack(c):
    return (c[:, 0] * _BIG + c[:, 1]) * _BIG + c[:, 2]


def _unpack(k):
    return torch.stack([k // (_BIG * _BIG), (k // _BIG) % _BIG, k % _BIG], 1)


def _root_limits(pos, levels):
    """the leaf range of the root: the lowest node that covers the points with their margins"""
    lo = (pos.min(0).values - 1.0).clamp_min(0.0).to(torch.int64).tolist()
    hi = (pos.max(0).values + 2.0).clamp_min(0.0).to(torch.int64).tolist()
    r = 1
    for ld in levels:
        r <<= ld
        if all(a // r == b // r for a, b in zip(lo, hi)):
            break
    b = 1 << levels[0]
    return [v // r * r // b for v in lo], [v // r * r // b + r // b for v in lo]


def _touched(pos, radius, up, levels, limits):
    """(leaves holding points, all leaves that the points' boxes [p - r, p + up r] touch), sorted"""
    b = 1 << levels[0]
    q = pos[(pos >= 0).all(1)]
    ip = q.to(torch.int64)
    c = ip // b
    held = torch.unique(_pack(c))
    if not radius > 0:
        return held, held
    lo = torch.div((ip.float() - radius).to(torch.int64), b, rounding_mode="trunc") - c
    hi = torch.div((ip.float() + up * radius).to(torch.int64), b, rounding_mode="trunc") - c
    keys = [held]
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                d = torch.tensor([dx, dy, dz], device=pos.device)
                m = ((lo <= d) & (hi >= d)).all(1)
                e = c[m] + d
                e = e[(e >= torch.tensor(limits[0], device=pos.device)).all(1) &
                      (e < torch.tensor(limits[1], device=pos.device)).all(1)]
                keys.append(torch.unique(_pack(e)))
    return held, torch.unique(torch.cat(keys))


def _full_bricks(pos, radius, levels):
    """leaf coordinates of a full build in pool order: leaves with points, then the dilation's"""
    held, every = _touched(pos, radius if radius >= 1.0 else 0.0, 2.0, levels, _root_limits(pos, levels))
    return _unpack(torch.cat([held, every[~torch.isin(every, held)]]))


_BRICKS = {}


def _brick_counts(case):
    """active bricks of each grid of the case, on the inputs of seed 0 (the other seeds' differ little)"""
    key = repr(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _BRICKS:
        k = case["kind"]
        if k == "sort":
            n = [0]
        elif k == "fusion":
            n = [len(_fused(_depth_frames(case, 0), LEVELS))]
        elif k == "batch":
            n = [len(_full_bricks(p, 1.0, LEVELS)) for p, _ in _clouds(case, 0)]
        else:
            inp = _inputs(case, 0)
            if k == "frame":
                n = [len(_full_bricks(inp["pos"], _topo_radius(case), (case["brick"],) + LEVELS[1:]))]
            elif k == "scatter":
                n = [len(_full_bricks(inp["pos"], case["radius"], LEVELS))]
            elif k == "surface":
                n = [_incremental(inp["pos"], case["radius"], LEVELS)[1]]
            elif k == "cloud":
                n = [len(_full_bricks((inp["q"].to(torch.int32) & 0xFFFF).float() * (case["extent"] / 65535.0), 2.0,
                                      LEVELS))]
            else:
                n = [len(_full_bricks(inp["pos"], 3.0, LEVELS))]
        _BRICKS[key] = n
    return _BRICKS[key]


def _layers(case):
    """layers of 16 x 16 bricks that each grid of the case reserves: its bricks and a little room"""
    return [-(-(n + n // 32 + 64) // 256) for n in _brick_counts(case)]


def _slots(used, layers):
    """bricks of the atlas (16 x 16 a layer): those reserved, or more when they do not suffice"""
    return max(layers, -(-used // 256)) * 256


class _Lookup:
    """leaf coordinates -> index in the list, -1 where there is none"""

    def __init__(self, bricks):
        self.lo = bricks.min(0).values - 1
        self.dim = bricks.max(0).values + 2 - self.lo
        self.table = torch.full((int(self.dim.prod()),), -1, dtype=torch.int32, device=bricks.device)
        self.table[self._index(bricks)] = torch.arange(len(bricks), dtype=torch.int32, device=bricks.device)

    def _index(self, c):
        r = c - self.lo
        return (r[:, 0] * self.dim[1] + r[:, 1]) * self.dim[2] + r[:, 2]

    def __call__(self, c):
        r = c - self.lo
        ok = ((r >= 0) & (r < self.dim)).all(1)
        return torch.where(ok, self.table[torch.where(ok, self._index(c), 0)].to(torch.int64), -1)


def _kernel64(d2, r):
    """M4 cubic spline of support r, normalised"""
    h = 0.5 * r
    q = d2.sqrt() / h
    w = torch.where(q < 1.0, 1.0 - 1.5 * q * q + 0.75 * q ** 3, 0.25 * (2.0 - q).clamp_min(0.0) ** 3)
    return w / (math.pi * h ** 3)


def _pairs(p, r, mode, look, b, chunk=500_000):
    """(point indices, flat interior voxel, p - v) of every point and voxel of its footprint in an active brick"""
    n = len(p)
    rmax = 1.0 if mode == "trilinear" else float(r.max())
    per = 2 if mode == "trilinear" else int(math.ceil(2.0 * rmax)) + 1
    for i0 in range(0, n, chunk):
        q = p[i0:i0 + chunk].double()
        live = (p[i0:i0 + chunk] >= 0).all(1)
        if mode == "trilinear":
            base = q.floor().to(torch.int64)
        else:
            base = (q - r[i0:i0 + chunk, None].double()).floor().to(torch.int64) + 1
        for kx in range(per):
            for ky in range(per):
                for kz in range(per):
                    v = base + torch.tensor([kx, ky, kz], device=p.device)
                    d = q - v
                    ok = live & (v >= 0).all(1)
                    if mode != "trilinear":
                        ok &= (d * d).sum(1) < r[i0:i0 + chunk].double() ** 2
                    vi, di = v[ok], d[ok]
                    slot = look(vi // b)
                    in_ = slot >= 0
                    l = vi % b
                    flat = ((slot * b + l[:, 2]) * b + l[:, 1]) * b + l[:, 0]
                    idx = torch.nonzero(ok)[:, 0][in_] + i0
                    yield idx, flat[in_], di[in_]


def _weights(idx, d, r, mode):
    if mode == "trilinear":
        return (1.0 - d.abs()).clamp_min(0.0).prod(1)
    return _kernel64((d * d).sum(1), r[idx].double())


def _splat64(p, w, r, mode, bricks, b, vel=None, into=None):
    """interior sums (bricks, b, b, b[, 3]) of the points' weights, or of weight * velocity"""
    n = len(p)
    if not torch.is_tensor(r):
        r = torch.full((n,), float(r), device=p.device)
    look = _Lookup(bricks)
    comps = 1 if vel is None else 3
    acc = torch.zeros((len(bricks) * b ** 3, comps), dtype=torch.float64, device=p.device)
    for idx, flat, d in _pairs(p, r, mode, look, b):
        k = _weights(idx, d, r, mode)
        if w is not None:
            k = k * w[idx].double()
        acc.index_add_(0, flat, k[:, None] if vel is None else k[:, None] * vel[idx].double())
    acc = acc.reshape((len(bricks), b, b, b) + ((3,) if vel is not None else ()))
    return acc if into is None else into + acc


def _neighbours(bricks):
    look = _Lookup(bricks)
    return {(dx, dy, dz): look(bricks + torch.tensor([dx, dy, dz], device=bricks.device))
            for dx in (-1, 0, 1) for dy in (-1, 0, 1) for dz in (-1, 0, 1)}


def _padded(inner, bricks, b, slots, bound=0.0, nbr=None):
    """the channel: every brick with its apron, copies of the neighbours' voxels or the boundary value"""
    P = b + 2
    tail = inner.shape[4:]
    out = torch.zeros((slots, P, P, P) + tail, dtype=inner.dtype, device=inner.device)
    nbr = nbr or _neighbours(bricks)
    dst = {-1: slice(0, 1), 0: slice(1, P - 1), 1: slice(P - 1, P)}
    src = {-1: slice(b - 1, b), 0: slice(0, b), 1: slice(0, 1)}
    m = len(bricks)
    for (dx, dy, dz), s in nbr.items():
        part = inner[:, src[dz], src[dy], src[dx]][s.clamp_min(0)]
        miss = (s < 0).reshape((-1,) + (1,) * (part.dim() - 1))
        out[:m, dst[dz], dst[dy], dst[dx]] = torch.where(miss, torch.full_like(part, bound), part)
    return out


def _smooth(chan, bricks, b, slots, bound, times):
    """(c + the six face neighbours) / 7 over the interiors, the aprons copied again after each time"""
    nbr = _neighbours(bricks)
    m = len(bricks)
    for _ in range(times):
        c = chan[:m]
        i = slice(1, b + 1)
        v = (c[:, i, i, i] + c[:, i, i, :-2] + c[:, i, i, 2:] + c[:, i, :-2, i] + c[:, i, 2:, i] + c[:, :-2, i, i] +
             c[:, 2:, i, i]) / 7.0
        chan = _padded(v, bricks, b, slots, bound, nbr)
    return chan


def _listed_min(p, radius, sc, bricks, b, chunk=500_000):
    """per interior voxel the smallest squared distance to the points listed in its subcell (p in 64 bits,
    listed by their 32-bit positions)"""
    pos32, p64 = p
    look = _Lookup(bricks)
    best = torch.full((len(bricks) * b ** 3,), 1e300, dtype=torch.float64, device=p64.device).view(torch.int64)
    o = torch.arange(sc, device=p64.device)
    off = torch.stack(torch.meshgrid(o, o, o, indexing="ij"), -1).reshape(-1, 3)
    reach = int(math.ceil((2.0 * radius + 1.0) / sc)) + 1
    for i0 in range(0, len(pos32), chunk):
        f, q = pos32[i0:i0 + chunk], p64[i0:i0 + chunk]
        lo = torch.div((f - radius).to(torch.int64), sc, rounding_mode="trunc") * sc
        hi = torch.div(((f + 1.0) + radius).to(torch.int64), sc, rounding_mode="trunc") * sc
        live = (f >= 0).all(1)
        for kx in range(reach):
            for ky in range(reach):
                for kz in range(reach):
                    s = lo + sc * torch.tensor([kx, ky, kz], device=f.device)
                    ok = live & (s <= hi).all(1) & (s >= 0).all(1)
                    s, qq = s[ok], q[ok]
                    slot = look(s // b)
                    s, qq, slot = s[slot >= 0], qq[slot >= 0], slot[slot >= 0]
                    for j in range(0, len(off), 32):
                        v = s[:, None, :] + off[None, j:j + 32, :]
                        d2 = ((qq[:, None, :] - v) ** 2).sum(2)
                        l = v % b
                        flat = ((slot[:, None] * b + l[..., 2]) * b + l[..., 1]) * b + l[..., 0]
                        best.scatter_reduce_(0, flat.reshape(-1), d2.reshape(-1).view(torch.int64), "amin")
    return best.view(torch.float64).reshape(len(bricks), b, b, b)


def _incremental(frames, radius, levels):
    """(bricks in slot order, most bricks of any step) of a full build and then incremental ones"""
    limits = _root_limits(frames[0], levels)
    pool = _pack(_full_bricks(frames[0], radius, levels))
    alive = torch.ones(len(pool), dtype=torch.bool, device=pool.device)
    most = len(pool)
    for pos in frames[1:]:
        _, every = _touched(pos, radius, 1.0, levels, limits)
        new = every[~torch.isin(every, pool[alive])]
        if len(new):
            alive = torch.cat([alive & torch.isin(pool, every), torch.ones(len(new), dtype=torch.bool,
                                                                         device=pool.device)])
            pool = torch.cat([pool, new])
        most = max(most, int(alive.sum()))
    return _unpack(pool[alive]), most


def _fused(frames, levels):
    limits = _root_limits(frames[0][0], levels)
    pool = _pack(_full_bricks(frames[0][0], 1.0, levels))
    for pos, _ in frames[1:]:
        _, every = _touched(pos, 1.0, 1.0, levels, limits)
        pool = torch.cat([pool, every[~torch.isin(every, pool)]])
    return _unpack(pool)


def _scatter64(pos, radius, bricks, b):
    """ScatterDensity: (1 - d^2 / r^2)^3 at a point's voxel and its six neighbours inside its own brick"""
    look = _Lookup(bricks)
    acc = torch.zeros(len(bricks) * b ** 3, dtype=torch.float64, device=pos.device)
    q = pos[(pos >= 0).all(1)]
    v0 = q.to(torch.int64)
    slot = look(v0 // b)
    for off in ((0, 0, 0), (-1, 0, 0), (1, 0, 0), (0, -1, 0), (0, 1, 0), (0, 0, -1), (0, 0, 1)):
        v = v0 + torch.tensor(off, device=pos.device)
        l = v - v0 // b * b
        ok = ((l >= 0) & (l < b)).all(1)
        c = ((v.double() - q.double()) ** 2).sum(1) / radius ** 2
        flat = ((slot * b + l[:, 2]) * b + l[:, 1]) * b + l[:, 0]
        acc.index_add_(0, flat[ok], ((1.0 - c) ** 3)[ok])
    return acc.reshape(len(bricks), b, b, b)


def _gradient64(p, w, r, grad, bricks, b):
    """adjoint of the cubic density splat: d/d(position, weight, radius) for dL/drho on the interiors"""
    look = _Lookup(bricks)
    n = len(p)
    flat_g = grad.reshape(-1)
    dp = torch.zeros((n, 3), dtype=torch.float64, device=p.device)
    dw, dr = torch.zeros(n, dtype=torch.float64, device=p.device), torch.zeros(n, dtype=torch.float64, device=p.device)
    for idx, flat, d in _pairs(p, r, "cubic", look, b):
        gv = flat_g[flat]
        wi, h = w[idx].double(), 0.5 * r[idx].double()
        dist = (d * d).sum(1).sqrt()
        q = dist / h
        norm = 1.0 / (math.pi * h ** 3)
        m4 = torch.where(q < 1.0, 1.0 - 1.5 * q * q + 0.75 * q ** 3, 0.25 * (2.0 - q) ** 3)
        dm = torch.where(q < 1.0, -3.0 * q + 2.25 * q * q, -0.75 * (2.0 - q) ** 2)
        s = torch.where(dist > 0, gv * wi * norm * dm / (h * dist.clamp_min(1e-300)), 0.0)
        dp.index_add_(0, idx, s[:, None] * d)
        dw.index_add_(0, idx, gv * norm * m4)
        dr.index_add_(0, idx, -gv * wi * norm * (3.0 * m4 + q * dm) / (2.0 * h))
    return dp, dw, dr


def exact(case, seed):
    k = case["kind"]
    if k == "sort":
        return None
    layers = _layers(case)[0]
    if k == "fusion":
        frames = _depth_frames(case, seed)
        bricks = _fused(frames, LEVELS)
        den = conf = None
        for pos, c in frames:
            den = _splat64(pos, None, 1.0, "trilinear", bricks, 8, into=den)
            conf = _splat64(pos, c, 1.0, "trilinear", bricks, 8, into=conf)
        s = _slots(len(bricks), layers)
        return {"density": _padded(den, bricks, 8, s).reshape(-1), "confidence": _padded(conf, bricks, 8, s).reshape(-1)}
    if k == "batch":
        out = []
        for (p, w), la in zip(_clouds(case, seed), _layers(case)):
            bricks = _full_bricks(p, 1.0, LEVELS)
            rho = _splat64(p, w, 1.0, "trilinear", bricks, 8)
            out.append(_padded(rho, bricks, 8, _slots(len(bricks), la)).reshape(-1))
        return out
    inp = _inputs(case, seed)
    if k == "frame":
        levels, b = (case["brick"],) + LEVELS[1:], 1 << case["brick"]
        bricks = _full_bricks(inp["pos"], _topo_radius(case), levels)
        s, nbr = _slots(len(bricks), layers), _neighbours(bricks)
        args = (inp["pos"], inp["w"], case["radius"], case["mode"], bricks, b)
        out = {"density": _padded(_splat64(*args), bricks, b, s, 0.0, nbr).reshape(-1)}
        if case["vel"]:
            v = _padded(_splat64(*args, vel=inp["vel"]), bricks, b, s, 0.0, nbr)
            out["velocity"] = torch.cat([v, torch.zeros_like(v[..., :1])], -1).reshape(-1)
        if case["source"] == "host":
            out["bricks"] = None
        return out
    if k == "scatter":
        bricks = _full_bricks(inp["pos"], case["radius"], LEVELS)
        d = _scatter64(inp["pos"], case["radius"], bricks, 8)
        return {"density": _padded(d, bricks, 8, _slots(len(bricks), layers)).reshape(-1), "colour": None}
    if k == "surface":
        bricks, most = _incremental(inp["pos"], case["radius"], LEVELS)
        p = inp["pos"][-1]
        dist = _listed_min((p, p.double()), case["radius"], case["subcell"], bricks, 8).sqrt()
        level = case["op"] == "levelset"
        bv = 3.0 if level else 0.0
        v = (dist - case["radius"]).clamp_max(3.0) if level else (case["radius"] - dist).clamp_min(0.0)
        s = _slots(most, layers)
        return {"surface": _smooth(_padded(v, bricks, 8, s, bv), bricks, 8, s, bv, 2).reshape(-1), "colour": None}
    if k == "cloud":
        d = torch.tensor(case["extent"] / 65535.0, dtype=torch.float32)
        pos = ((inp["q"].to(torch.int32) & 0xFFFF).double() * float(d)).float()
        bricks = _full_bricks(pos, 2.0, LEVELS)
        # the lists keep 16-bit fractions of the points' box, formed in single precision
        lo = (pos.min(0).values - 1.0).clamp_min(0.0)
        rg = (pos.max(0).values + 2.0).clamp_min(0.0) - lo
        q = ((pos - lo) / rg * 65535.0).clamp(0.0, 65535.0).floor().double()
        p64 = q / 65535.0 * rg.double() + lo.double()
        v = (_listed_min((pos, p64), 1.0, 4, bricks, 8).sqrt() - 1.0).clamp_max(3.0)
        s = _slots(len(bricks), layers)
        return {"levelset": _smooth(_padded(v, bricks, 8, s, 3.0), bricks, 8, s, 3.0, 1).reshape(-1)}
    # gradient
    bricks = _full_bricks(inp["pos"], 3.0, LEVELS)
    s, nbr = _slots(len(bricks), layers), _neighbours(bricks)
    target = _padded(_splat64(inp["other"], inp["w"], inp["r"], "cubic", bricks, 8), bricks, 8, s, 0.0, nbr).float()
    rho = _splat64(inp["pos"], inp["w"], inp["r"], "cubic", bricks, 8)
    inner = target[:len(bricks), 1:9, 1:9, 1:9].double()
    dp, dw, dr = _gradient64(inp["pos"], inp["w"], inp["r"], 2.0 * (rho - inner), bricks, 8)
    return {"density": _padded(rho, bricks, 8, s, 0.0, nbr).reshape(-1), "dpos": dp, "dweight": dw, "dradius": dr}


# --------------------------------------------------------------------------- work

def work(case):
    """bytes: every input read once and every output written once; flops: the voxel updates"""
    k, n = case["kind"], case.get("n")
    if k == "sort":
        return {"bytes": 16.0 * n, "flops": 0.0}
    nb = sum(_brick_counts(case))
    if k == "fusion":
        n = sum(len(p) for p, _ in _depth_frames(case, 0))
        return {"bytes": 16.0 * n + 8000.0 * nb, "flops": 2 * 8 * 6.0 * n}
    if k == "batch":
        n = sum(_cloud_sizes(case))
        return {"bytes": 16.0 * n + 4000.0 * nb, "flops": 8 * 6.0 * n}
    if k == "frame":
        b = 1 << case["brick"]
        vox = 8.0 if case["mode"] == "trilinear" else 4.0 / 3.0 * math.pi * case["radius"] ** 3
        per = 12 + (12 if case["vel"] else 0) + (4 if case["weight"] else 0)
        return {"bytes": float(per) * n + nb * (b + 2.0) ** 3 * (20 if case["vel"] else 4),
                "flops": n * vox * (6.0 if case["mode"] == "trilinear" else 20.0 + (6.0 if case["vel"] else 0.0))}
    if k == "scatter":
        return {"bytes": 16.0 * n + 8000.0 * nb, "flops": 7 * 12.0 * n}
    if k == "surface":
        return {"bytes": case["steps"] * 16.0 * n + 8000.0 * nb,
                "flops": case["steps"] * (n * 4.2 * 8.0 + 2 * 8 * 512.0 * nb)}
    if k == "cloud":
        return {"bytes": 6.0 * n + 4000.0 * nb, "flops": n * 4.2 * 8.0 + 8 * 512.0 * nb}
    mean = 4.0 / 3.0 * math.pi * (case["rmin"] + case["rmax"]) * (case["rmin"] ** 2 + case["rmax"] ** 2) / 4.0
    return {"bytes": (20.0 + 20.0) * n + 8000.0 * nb, "flops": n * mean * (20.0 + 45.0)}
