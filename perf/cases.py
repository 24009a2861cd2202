"""Timed cases of the framework's work: frames of the five traversals, batched
and served frames, and octree builds, each through a public entry point.

A case names a workload (``kind``), a volume and its size, and the options of
the call.  The volumes are the repository's synthetic stand-ins
(``xenodon_gb300.volumes``): Gaussian blobs, a CT-scan-shaped shell and a
cosmology-like gas field.
"""
import ctypes
import math
import random

import numpy as np
import torch

import xenodon_gb300 as xg
from xenodon_gb300 import cameras, volumes

_CTX = None


def _context():
    """The one device context a program of this framework holds."""
    global _CTX
    if _CTX is None:
        _CTX = xg.Context(0)
    return _CTX


# ------------------------------------------------------------------- cases ---

def listed():
    return [
        # a thumbnail or interactive preview of a small octree into host
        # memory: the smallest call, bound by launch and read-back latency
        {"name": "host-thumb-rope", "kind": "host", "volume": "blobs", "dx": 64, "dy": 64, "dz": 64,
         "traversal": "svo-rope", "w": 160, "h": 120, "view": "outside", "emission": False},
        # the 128^3 grid at 512x512 with the float emission beside the image
        # (tone mapping or numeric use of the result)
        {"name": "dda-blobs-512", "kind": "frame", "volume": "blobs", "dx": 128, "dy": 128, "dz": 128,
         "traversal": "dda", "w": 512, "h": 512, "view": "outside", "emission": True},
        # a UHD frame of a large simulation grid: the largest plain DDA frame
        {"name": "dda-gas-4k", "kind": "frame", "volume": "gas", "dx": 1024, "dy": 1024, "dz": 1024,
         "traversal": "dda", "w": 3840, "h": 2160, "view": "outside", "emission": False},
        # frames of the CT scan's octree along its camera path, HD: outside
        # (orbit) and inside the volume
        {"name": "naive-ct-1080p", "kind": "frame", "volume": "ct", "dx": 512, "dy": 361, "dz": 512,
         "traversal": "svo-naive", "w": 1920, "h": 1080, "view": "outside", "emission": False},
        {"name": "df-ct-1080p", "kind": "frame", "volume": "ct", "dx": 512, "dy": 361, "dz": 512,
         "traversal": "svo-df", "w": 1920, "h": 1080, "view": "outside", "emission": True},
        {"name": "rope-ct-inside-1080p", "kind": "frame", "volume": "ct", "dx": 512, "dy": 361, "dz": 512,
         "traversal": "svo-rope", "w": 1920, "h": 1080, "view": "inside", "emission": False},
        # a UHD frame of the large simulation's octree
        {"name": "esvo-gas-4k", "kind": "frame", "volume": "gas", "dx": 1024, "dy": 1024, "dz": 1024,
         "traversal": "esvo", "w": 3840, "h": 2160, "view": "outside", "emission": False},
        # many small frames from all around a volume in one batched launch
        # (turntables, training views)
        {"name": "batch-gas-256", "kind": "batch", "volume": "gas", "dx": 512, "dy": 512, "dz": 512,
         "traversal": "esvo+svo-df+svo-rope", "frames": 48, "w": 256, "h": 256},
        # an octree built on the device for rendering, then its first frame
        {"name": "build-gas-1024", "kind": "build", "volume": "gas", "dx": 1024, "dy": 1024, "dz": 1024,
         "svo_type": "sparse", "lean": True, "heuristic": "chan-diff", "threshold": 0.0,
         "traversal": "esvo", "w": 640, "h": 360},
        # the same with ropes, from a CT-scan-shaped grid of odd size
        {"name": "build-ct-rope", "kind": "build", "volume": "ct", "dx": 509, "dy": 361, "dz": 487,
         "svo_type": "rope", "lean": False, "heuristic": "chan-diff", "threshold": 0.0,
         "traversal": "svo-rope", "w": 640, "h": 360},
        # `convert`: a grid in host memory to the reference's node array in
        # host memory, nodes merged into a DAG
        {"name": "convert-ct-dag", "kind": "convert", "volume": "ct", "dx": 203, "dy": 143, "dz": 197,
         "svo_type": "dag", "heuristic": "std-dev", "threshold": 2.0},
        # a small device grid rebuilt in a loop without allocation (edited or
        # simulated volumes)
        {"name": "static-blobs-rope", "kind": "static", "volume": "blobs", "dx": 96, "dy": 96, "dz": 96,
         "svo_type": "rope", "heuristic": "chan-diff", "threshold": 0.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_dims(rng, lo, hi):
    """A volume kind and its size: cubic for blobs and gas, any box for CT."""
    vol = rng.choice(["blobs", "ct", "ct", "gas"])
    if vol == "blobs":
        n = _log(rng, min(lo, 160), min(hi, 160))
        return vol, n, n, n
    if vol == "gas":
        n = _log(rng, lo, hi)
        return vol, n, n, n
    n = _log(rng, lo, hi)
    return (vol,) + tuple(max(8, int(n * rng.uniform(0.6, 1.0))) for _ in range(3))


def draw(rng):
    kind = rng.choice(["host", "frame", "frame", "frame", "batch", "build", "build", "convert", "static"])
    if kind in ("host", "frame"):
        trav = rng.choice(["dda", "svo-naive", "esvo", "svo-df", "svo-rope"])
        vol, dx, dy, dz = _draw_dims(rng, 48, 640)
        px = _log(rng, 96 * 96, 1920 * 1080) if kind == "frame" else _log(rng, 96 * 96, 1280 * 720)
        w = max(16, int(math.sqrt(px * rng.uniform(0.8, 2.0))))
        return {"kind": kind, "volume": vol, "dx": dx, "dy": dy, "dz": dz, "traversal": trav, "w": w,
                "h": max(16, px // w), "view": rng.choice(["outside", "inside"]), "emission": rng.random() < 0.3}
    if kind == "batch":
        vol, dx, dy, dz = _draw_dims(rng, 64, 512)
        side = _log(rng, 64, 384)
        trav = rng.choice(["dda", "esvo", "svo-naive+svo-df", "esvo+svo-rope", "svo-naive+esvo+svo-df+svo-rope"])
        return {"kind": kind, "volume": vol, "dx": dx, "dy": dy, "dz": dz, "traversal": trav,
                "frames": rng.randint(4, 64), "w": side, "h": max(16, int(side * rng.uniform(0.6, 1.0)))}
    heur = rng.choice(["chan-diff", "chan-diff", "std-dev"])
    thr = float(rng.choice([0, 0, 4, 16])) if heur == "chan-diff" else rng.choice([0.5, 2.0, 6.5])
    case = {"kind": kind, "svo_type": rng.choice(["sparse", "dag", "rope"]), "heuristic": heur, "threshold": thr}
    if kind == "build":
        vol, dx, dy, dz = _draw_dims(rng, 48, 640)
        case["lean"] = rng.random() < 0.4
        if case["lean"]:
            case["svo_type"] = "sparse"
        case["traversal"] = "svo-rope" if case["svo_type"] == "rope" else rng.choice(["svo-naive", "esvo", "svo-df"])
        case["w"], case["h"] = 640, 360
    elif kind == "convert":
        vol, dx, dy, dz = _draw_dims(rng, 32, 200)
    else:
        vol, dx, dy, dz = _draw_dims(rng, 16, 96)
        if case["svo_type"] == "dag":  # its tables share the fixed scratch
            vol, dx, dy, dz = _draw_dims(rng, 16, 48)
    return {**case, "volume": vol, "dx": dx, "dy": dy, "dz": dz}


# ----------------------------------------------------------------- volumes ---

def _grid(case, seed, host):
    """The case's RGBA8 grid, (dz, dy, dx, 4): numpy when `host`, else a tensor
    on the GPU."""
    if case["volume"] == "gas":
        g = volumes.gas_field(case["dx"], seed=seed, device="cuda", as_tensor=not host)
    elif case["volume"] == "ct":
        g = volumes.ct_shell(case["dx"], case["dy"], case["dz"], seed=seed, device="cuda")
    else:
        g = volumes.blobs(case["dx"], seed=seed)
    if not host and isinstance(g, np.ndarray):
        g = torch.from_numpy(g).cuda()
    torch.cuda.synchronize()
    return g


def _dims(case):
    return case["dx"], case["dy"], case["dz"]


def _side(case):
    return 1 << (max(_dims(case)) - 1).bit_length()


def _centre(case, trav):
    """The grid's centre in camera units: a grid spans [0, dim/max_dim], an
    octree [0, 1] with the grid in its low corner."""
    unit = max(_dims(case)) if trav == "dda" else _side(case)
    return np.array([d / unit for d in _dims(case)]) * 0.5


def _camera(case, trav, seed, k=0, n=1):
    rng = random.Random(seed * 7919 + k)
    c = _centre(case, trav)
    extent = 2.0 * float(c.max())
    if case.get("view") == "inside":
        a = rng.uniform(0.0, 2.0 * math.pi)
        pos = c + extent * np.array([0.05, 0.02, -0.1])
        return cameras.look_at(pos, pos + np.array([math.sin(a), 0.1, math.cos(a)]))
    if n > 1:
        return cameras.fibonacci_sphere(n, c, 1.8 * extent,
                                        cameras.forward_length_for_vfov(45.0, case["w"], case["h"]))[k]
    a = rng.uniform(0.0, 2.0 * math.pi)
    pos = c + extent * rng.uniform(1.4, 1.8) * np.array([math.sin(a), rng.uniform(-0.3, 0.3), -math.cos(a)])
    return cameras.look_at(pos, c)


def _coefficient(case):
    return 10.0 if case["volume"] == "ct" else 2.0


def _params(case):
    return xg.make_params(case["w"], case["h"], _coefficient(case))


def _most_nodes(case):
    """The nodes of the largest tree over a grid of this size: the root and,
    per depth, the eight children of every cell that touches the grid."""
    n, e = 1, 1
    while e < _side(case):
        e *= 2
        n += 8 * math.prod(-(-d // e) for d in _dims(case))
    return n


class _Released:
    """Holds volumes and gives their device memory back with itself."""

    def __init__(self):
        self.volumes = []

    def add(self, vol):
        self.volumes.append(vol)
        return vol

    def __del__(self):
        for v in self.volumes:
            v.release()


def _volume(case, seed, trav, keep):
    ctx = _context()
    g = _grid(case, seed, host=False)
    if trav == "dda":
        vol = ctx.upload_grid_device(g.data_ptr(), _dims(case))
    elif trav == "svo-rope" or "svo-rope" in trav.split("+"):
        vol, _ = ctx.build_svo_volume(g.data_ptr(), _dims(case), "rope")
    else:
        vol, _ = ctx.build_svo_volume(g.data_ptr(), _dims(case), "sparse", lean=True)
    return keep.add(vol)


# ---------------------------------------------------------------- the calls ---

def prepare(case, seed):
    keep = _Released()
    s = {"case": case, "keep": keep}
    kind = case["kind"]
    if kind in ("host", "frame"):
        s["vol"] = _volume(case, seed, case["traversal"], keep)
        s["camera"] = xg.make_camera(*_camera(case, case["traversal"], seed))
        s["params"] = _params(case)
        if kind == "host":
            s["out"] = np.empty((case["h"], case["w"], 4), np.uint8)
        else:
            s["rgba"] = torch.empty((case["h"], case["w"], 4), dtype=torch.uint8, device="cuda")
            if case["emission"]:
                s["emission"] = torch.empty((case["h"], case["w"], 3), dtype=torch.float32, device="cuda")
    elif kind == "batch":
        vol = _volume(case, seed, case["traversal"], keep)
        travs = case["traversal"].split("+")
        n = case["frames"]
        s["rgba"] = torch.empty((n, case["h"], case["w"], 4), dtype=torch.uint8, device="cuda")
        s["specs"] = []
        for k in range(n):
            t = travs[k % len(travs)]
            cam = xg.make_camera(*_camera(case, t, seed, k, n))
            s["specs"].append((vol, t, cam, _params(case), s["rgba"][k].data_ptr()))
    elif kind == "build":
        s["grid"] = _grid(case, seed, host=False)
        s["camera"] = xg.make_camera(*_camera(case, case["traversal"], seed))
        s["params"] = _params(case)
        s["rgba"] = torch.empty((case["h"], case["w"], 4), dtype=torch.uint8, device="cuda")
    elif kind == "convert":
        _context()
        s["grid"] = _grid(case, seed, host=True)
        s["nodes"] = np.zeros((_most_nodes(case), 10), np.int32)  # the program's own tree
    else:
        s["grid"] = _grid(case, seed, host=False)
        s["nodes"] = torch.zeros((_most_nodes(case), 10), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "host":
        rgba, emission, _ = _context().render(state["vol"], case["traversal"], state["camera"], state["params"],
                                              emission=case["emission"], out=state["out"])
        return [rgba, emission] if case["emission"] else [rgba]
    if kind == "frame":
        em = state.get("emission")
        _context().render_device(state["vol"], case["traversal"], state["camera"], state["params"],
                                 state["rgba"].data_ptr(), em.data_ptr() if em is not None else None, None, stream)
        return [state["rgba"], em] if em is not None else [state["rgba"]]
    if kind == "batch":
        ctx = _context()
        jobs = ctx.make_jobs(state["specs"])
        ctx.render_batch(jobs, len(state["specs"]), None, stream)
        return [state["rgba"]]
    if kind == "build":
        ctx = _context()
        vol, stats = ctx.build_svo_volume(state["grid"].data_ptr(), _dims(case), case["svo_type"], case["heuristic"],
                                          case["threshold"], lean=case["lean"])
        ctx.render_device(vol, case["traversal"], state["camera"], state["params"], state["rgba"].data_ptr(),
                          None, None, stream)
        torch.cuda.current_stream().synchronize()  # the frame has to be done before its volume goes
        vol.release()
        return {"rgba": state["rgba"], "stats": stats}
    if kind == "convert":
        nodes, stats = _context().build_svo(state["grid"], case["svo_type"], case["heuristic"], case["threshold"])
        state["nodes"][:len(nodes)] = nodes.view(np.int32)
        return {"nodes": state["nodes"], "stats": stats}
    lib = xg.load_library()
    st = xg.BuildStats()
    r = lib.xn_build_svo_static(state["grid"].data_ptr(), *_dims(case), xg.SVO_TYPES[case["svo_type"]],
                                xg.HEURISTICS[case["heuristic"]], case["threshold"], state["nodes"].data_ptr(),
                                state["nodes"].shape[0], ctypes.byref(st), stream)
    if r != xg.XN_OK:
        raise xg.XenodonError(r, lib.xn_last_error().decode())
    return {"nodes": state["nodes"], "stats": {f: int(getattr(st, f)) for f, _ in st._fields_}}


# --------------------------------------------------------------------- work ---

def work(case):
    """Bytes: each input and output once (a frame reads at most the volume's
    voxels; a build reads the grid and writes at least one 40-byte node, or 36
    bytes of the device layout, per eight voxels).  Operations: a ray's steps
    at one voxel each and about 20 operations a step; a build compares and
    sums four channels of every voxel."""
    voxels = math.prod(_dims(case))
    if case["kind"] in ("host", "frame", "batch"):
        rays = case["w"] * case["h"] * case.get("frames", 1)
        out = rays * (16 if case.get("emission") else 4)
        steps = 0.3 * sum(_dims(case)) / 3.0
        return {"bytes": 4.0 * min(voxels, rays * steps) + out, "flops": rays * steps * 20.0}
    per_voxel = 4.0 + (36.0 if case.get("lean") else 40.0) / 8.0
    return {"bytes": voxels * per_voxel, "flops": voxels * 12.0}


# -------------------------------------------------------------------- exact ---

def exact(case, seed):
    """The emission of every ray in 64 bits: the sum over the voxels that the
    ray crosses of colour/255 times the length inside, times the coefficient.
    All five traversals compute this integral (an octree merges equal voxels
    only); images, node arrays and counts are whole numbers."""
    if case["kind"] not in ("host", "frame") or not case["emission"]:
        return None
    trav = case["traversal"]
    g = _grid(case, seed, host=False)
    unit = float(max(_dims(case)) if trav == "dda" else _side(case))
    forward, up, pos = (np.float32(v).astype(np.float64) for v in _camera(case, trav, seed))
    w, h = case["w"], case["h"]
    f64 = {"dtype": torch.float64, "device": "cuda"}

    def unit_vector(v):
        return v / np.linalg.norm(v)

    right = unit_vector(np.cross(up, forward))
    down = unit_vector(np.cross(right, forward))
    u = torch.arange(w, **f64)[None, :] / w - 0.5
    v = (torch.arange(h, **f64)[:, None] / h - 0.5) * (h / w)
    rd = torch.stack([(right[k] * u + down[k] * v + forward[k]).expand(h, w) for k in range(3)], -1).reshape(-1, 3)
    rd = rd / rd.norm(dim=1, keepdim=True)
    rd = torch.where(rd.abs() < 2.0 ** -23, torch.full_like(rd, 2.0 ** -23), rd)
    dims = torch.tensor(_dims(case), **f64)
    ro = torch.tensor(pos, **f64) * unit
    t0, t1 = (0.0 - ro) / rd, (dims - ro) / rd
    enter = torch.minimum(t0, t1).amax(1).clamp_min(0.0)
    leave = torch.maximum(t0, t1).amin(1)
    live = torch.nonzero(enter < leave).reshape(-1)
    total = torch.zeros((rd.shape[0], 3), **f64)
    rd, t, leave = rd[live], enter[live], leave[live]
    texels = g.reshape(-1, 4)[:, :3]
    sgn = torch.where(rd > 0, 1, -1)
    # the cell of the first point inside, and the parameter of its far planes
    mid = ro + rd * t[:, None]
    cell = torch.minimum(torch.floor(mid).clamp_min(0.0), dims - 1).to(torch.int64)
    far = ((cell + (sgn > 0)).to(torch.float64) - ro) / rd
    acc = torch.zeros((rd.shape[0], 3), **f64)
    step = (1.0 / rd).abs()
    dx, dy, dz = _dims(case)
    lim = torch.tensor(_dims(case), device="cuda")
    for i in range(dx + dy + dz + 3):
        nxt, axis = far.min(1)
        nxt = torch.minimum(nxt, leave)
        inside = ((cell >= 0) & (cell < lim)).all(1)
        idx = torch.where(inside, cell[:, 0] + dx * (cell[:, 1] + dy * cell[:, 2]), 0)
        length = torch.where(inside, (nxt - t).clamp_min(0.0), 0.0)
        acc += texels[idx].to(torch.float64) * length[:, None]
        t = torch.maximum(t, nxt)
        one = torch.nn.functional.one_hot(axis, 3)
        cell = cell + sgn * one
        far = far + step * one
        if i % 64 == 63 and not bool((t < leave).any()):
            break
    total[live] = acc * (_coefficient(case) / 255.0 / unit)
    return [None, total.reshape(h, w, 3)]
