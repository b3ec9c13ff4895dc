"""Performance cases: the work a program has this framework do, through the
package's public entry points.

Three groups:
- frames: one RenderFrame of a resident scene (the per-frame loop's main path),
  one RenderFrame of a camera in motion whose blocks stream through a cache
  smaller than the scene, one RenderViews of many views, one round of a
  RenderServer's clients;
- the feedback primitives GPUSort and GPUScan on device arrays;
- feedback_unique on a frame's (or many frames') feedback words.

Scenes are the builder's seeded terrains, written once per machine to the
temporary directory; cameras, keys and words come from the seed.
"""
import math
import os
import random
import tempfile

import numpy as np
import torch

import rayt_gb300 as R

NO_HIT = 0x7FFFFFFF

# name: depth, nodes in a block, sphere shells, largest radius.  t8 is the
# smoke test's scene, t10 the 512x512 benchmark's; t11 stands for the
# flythrough scenes (terrain and many shells, 0.7 GB of blocks).
SCENES = {"t8": (8, 512, 60, 24), "t10": (10, 4096, 0, 256), "t11": (11, 4096, 500, 128)}
BLOCKS = {"t8": 793, "t10": 758, "t11": 13831}
VIEW_SIZES = [(256, 256), (640, 480), (1280, 720), (1920, 1080)]
CLIENT_SIZES = [(1280, 720), (1920, 1080), (2560, 1440)]
LOOP = 32  # frames of the moving camera's closed path

_loaders = {}


def _loader(scene):
    """The opened block file of a scene, built when the machine has none yet."""
    if scene not in _loaders:
        depth, nib, spheres, radius = SCENES[scene]
        folder = os.path.join(tempfile.gettempdir(), "rayt_perf_%d" % os.getuid())
        os.makedirs(folder, exist_ok=True)
        path = os.path.join(folder, "d%d_n%d_s%d_r%d.tree" % (depth, nib, spheres, radius))
        if not os.path.exists(path):
            part = "%s.%d" % (path, os.getpid())
            R.build_terrain(part, depth, nib, spheres=spheres, min_radius=2 if depth < 10 else 8, max_radius=radius)
            os.replace(part, path)
        _loaders[scene] = R.StoredOctreeLoader(path)
    return _loaders[scene]


def _cache(scene, blocks=0):
    c = R.GPUOctreeCacheManager(blocks, _loader(scene))
    c.InitialFillCache()
    return c


def _camera(rng, w, h):
    """A camera over the terrain, looking 15 to 35 degrees down."""
    pos = (rng.uniform(0.15, 0.85), rng.uniform(0.62, 0.85), rng.uniform(0.15, 0.85))
    return R.Camera(rng.uniform(0, 360), rng.uniform(-35, -15), 0.0, pos, 60.0, w / h).view_proj_inv()


def _loop_cameras(rng, w, h):
    """A closed round flight of LOOP frames, looking ahead and 25 degrees down."""
    r, a0, y = 0.2, rng.uniform(0, 2 * math.pi), rng.uniform(0.66, 0.8)
    cx, cz = rng.uniform(0.35, 0.65), rng.uniform(0.35, 0.65)
    out = []
    for i in range(LOOP):
        a = a0 + 2 * math.pi * i / LOOP
        pos = (cx + r * math.cos(a), y, cz + r * math.sin(a))
        yaw = math.degrees(math.atan2(-math.sin(a), -math.cos(a)))
        out.append(R.Camera(yaw, -25.0, 0.0, pos, 60.0, w / h).view_proj_inv())
    return out


class _Device:
    """A device buffer of the library as the array interface torch reads; the
    tensor holds this object, and so the renderer that owns the buffer."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _tensor(owner, ptr, shape, typestr):
    return torch.as_tensor(_Device(owner, ptr, shape, typestr), device="cuda")


class _HostImage(np.ndarray):
    """A client's host image that holds the server that owns it."""

    owner = None


def _sizes(case, pool):
    """The sizes of a case's views or clients: a fixed draw from the pool."""
    rng = random.Random(case["sizes"])
    return [rng.choice(pool) for _ in range(case["count"])]


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _keys(case, seed):
    """int32 keys: anything, values of a small range around zero, or block IDs."""
    lo, hi = {"wide": (-2 ** 31, 2 ** 31 - 1), "narrow": (-100, 101), "blocks": (0, 1 << 24)}[case["keys"]]
    return torch.randint(lo, hi, (case["n"],), dtype=torch.int32, device="cuda", generator=_gen(seed))


def _words(case, seed):
    """Feedback words of a pass: NO_HIT but for a share `kept`, of which half
    are faults (-block - 1) and half hits ((node + 1) << 1 | dup), the blocks
    Zipf(1.1) over [0, blocks)."""
    n, blocks, nib = case["n"], case["blocks"], case["nib"]
    g = _gen(seed)
    at = torch.nonzero(torch.rand(n, device="cuda", generator=g) < case["kept"]).view(-1)
    m = at.numel()
    u = torch.rand(m, device="cuda", generator=g, dtype=torch.float64)
    ids = ((1.0 + u * (blocks ** -0.1 - 1.0)) ** -10.0).to(torch.int64).sub_(1).clamp_(0, blocks - 1)
    del u
    node = ids if nib == 0 else ids * nib + torch.randint(0, nib, (m,), device="cuda", generator=g)
    dup = torch.randint(0, 2, (m,), device="cuda", generator=g)
    hit = ((node + 1) << 1) | dup
    fault = torch.randint(0, 2, (m,), device="cuda", generator=g, dtype=torch.bool)
    out = torch.full((n,), NO_HIT, dtype=torch.int32, device="cuda")
    out[at] = torch.where(fault, -ids - 1, hit).to(torch.int32)
    return out


def listed():
    return [
        # a preview or thumbnail: what a call costs when the GPU has little to do
        {"name": "frame_128x96", "kind": "frame", "scene": "t8", "width": 128, "height": 96, "lod": 1.0, "depth": False},
        # an interactive window of the reference's size over a resident scene
        {"name": "frame_512x512", "kind": "frame", "scene": "t10", "width": 512, "height": 512, "lod": 1.0, "depth": False},
        # a full-screen frame of a ragged size, with depth and hit nodes for a
        # compositor, at the reference's default voxel size
        {"name": "frame_1919x1079_depth", "kind": "frame", "scene": "t11", "width": 1919, "height": 1079, "lod": 1.5,
         "depth": True},
        # a flight through a scene larger than the cache, frames delivered to
        # host memory: several passes and block uploads in every frame
        {"name": "stream_1280x720", "kind": "stream", "scene": "t11", "width": 1280, "height": 720, "lod": 1.0,
         "blocks": 1600},
        # many views at once: thumbnails to full-screen ones in one call
        {"name": "views_12", "kind": "views", "scene": "t11", "count": 12, "sizes": 7, "lod": 1.0},
        # a service: a frame for each of several clients, delivered to the host
        {"name": "served_8", "kind": "served", "scene": "t11", "count": 8, "sizes": 100, "lod": 1.0},
        # the size and values of the reference's own sort test: all latency
        {"name": "sort_2013", "kind": "sort", "n": 2013, "keys": "narrow"},
        # an offline sort of many keys
        {"name": "sort_64m", "kind": "sort", "n": 1 << 26, "keys": "wide"},
        # offsets of a frame-sized list
        {"name": "scan_1000003", "kind": "scan", "n": 1000003},
        # offsets of a large list: all bandwidth
        {"name": "scan_256m", "kind": "scan", "n": 1 << 28},
        # the request list of one 1080p pass: most pixels hit
        {"name": "unique_frame", "kind": "unique", "n": 1920 * 1080, "kept": 0.7, "blocks": 1 << 15, "nib": 4096},
        # the feedback microbenchmark: 2^28 words, a tenth kept
        {"name": "unique_256m", "kind": "unique", "n": 1 << 28, "kept": 0.1, "blocks": 1 << 24, "nib": 0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "stream", "views", "served", "sort", "scan", "unique"])
    lod = round(rng.uniform(1.0, 2.0), 2)
    if kind == "frame":
        w = _log(rng, 64, 2560)
        return {"kind": kind, "scene": rng.choice(["t8", "t10", "t11"]), "width": w,
                "height": max(48, int(w / rng.uniform(1.0, 1.9))), "lod": lod, "depth": rng.random() < 0.3}
    if kind == "stream":
        w = _log(rng, 320, 1920)
        return {"kind": kind, "scene": "t11", "width": w, "height": int(w / rng.uniform(1.2, 1.9)), "lod": lod,
                "blocks": _log(rng, 1000, 2000)}
    if kind == "views":
        return {"kind": kind, "scene": rng.choice(["t10", "t11"]), "count": rng.randint(2, 16),
                "sizes": rng.randrange(1000), "lod": lod}
    if kind == "served":
        return {"kind": kind, "scene": rng.choice(["t10", "t11"]), "count": rng.randint(2, 8),
                "sizes": rng.randrange(1000), "lod": lod}
    if kind == "sort":
        return {"kind": kind, "n": _log(rng, 256, 1 << 26), "keys": rng.choice(["wide", "narrow", "blocks"])}
    if kind == "scan":
        return {"kind": kind, "n": _log(rng, 256, 1 << 28)}
    nib = rng.choice([0, 4096])
    return {"kind": kind, "n": _log(rng, 1024, 1 << 28), "kept": round(rng.uniform(0.05, 0.9), 2),
            "blocks": _log(rng, 1 << 10, 1 << 17 if nib else 1 << 28), "nib": nib}


def prepare(case, seed):
    kind, rng = case["kind"], random.Random(seed)
    s = {"kind": kind}
    if kind == "sort":
        s["src"] = _keys(case, seed)
        s["x"] = torch.empty_like(s["src"])
    elif kind == "scan":
        s["x"] = _keys(dict(case, keys="wide"), seed)
    elif kind == "unique":
        s["words"] = _words(case, seed)
        s["nib"] = case["nib"]
        s["out"] = torch.zeros_like(s["words"])
    elif kind in ("frame", "stream"):
        w, h = case["width"], case["height"]
        s["cache"] = _cache(case["scene"], case.get("blocks", 0))
        rt = s["renderer"] = R.GPURayTracer(s["cache"], w, h)
        rt.set_lod_voxel_size(case["lod"])
        rt.set_frame_time_limit(1e30)
        rt.seed(seed & 0xFFFFFFFF)
        if kind == "stream":
            s["image"] = torch.zeros((h, w, 4), dtype=torch.uint8, pin_memory=True)
            rt.set_host_image(s["image"].data_ptr(), s["image"].numel())
            s["cameras"], s["at"] = _loop_cameras(rng, w, h), 0
            for m in s["cameras"]:  # the flight is under way
                rt.RenderFrame(m)
        else:
            s["camera"] = _camera(rng, w, h)
            rt.set_depth_output(case["depth"])
            s["out"] = {"image": _tensor(rt, rt.out_image_device_ptr(), (h, w, 4), "|u1")}
            if case["depth"]:
                depth, nodes = rt.depth_device_ptrs()
                s["out"].update(depth=_tensor(rt, depth, (h, w), "<f4"), nodes=_tensor(rt, nodes, (h, w), "<i4"))
    elif kind == "views":
        sizes = _sizes(case, VIEW_SIZES)
        s["cache"] = _cache(case["scene"])
        rt = s["renderer"] = R.GPURayTracer.views(s["cache"], sizes)
        rt.set_lod_voxel_size(case["lod"])
        rt.set_frame_time_limit(1e30)
        rt.seed(seed & 0xFFFFFFFF)
        s["cameras"] = [_camera(rng, w, h) for w, h in sizes]
        s["out"] = [_tensor(rt, rt.out_image_device_ptr(v), (h, w, 4), "|u1") for v, (w, h) in enumerate(sizes)]
    elif kind == "served":
        sizes = _sizes(case, CLIENT_SIZES)
        pixels = sum(w * h + 64 for w, h in sizes)
        s["cache"] = _cache(case["scene"])
        sv = s["server"] = R.RenderServer(s["cache"], len(sizes), 4 * pixels, pixels, lod_voxel_size=case["lod"],
                                          deliver_to_host=True)
        sv.seed(seed & 0xFFFFFFFF)
        s["clients"] = [(sv.add_client(w, h), _camera(rng, w, h)) for w, h in sizes]
        s["out"] = [sv.host_image(c).view(_HostImage) for c, _ in s["clients"]]
        for image in s["out"]:
            image.owner = sv
    else:
        raise ValueError(kind)
    return s


def run(s):
    kind = s["kind"]
    if kind == "sort":  # in place, so each pass sorts a fresh copy
        s["x"].copy_(s["src"])
        R.GPUSort(s["x"], s["x"].numel())
        return s["x"]
    if kind == "scan":  # in place; any int32 values are an input
        R.GPUScan(s["x"], s["x"].numel())
        return s["x"]
    if kind == "unique":
        n = R.feedback_unique(s["words"], s["words"].numel(), s["nib"], s["out"])
        return {"count": n, "unique": s["out"]}
    if kind == "frame":
        s["renderer"].RenderFrame(s["camera"])
        return s["out"]
    if kind == "stream":  # the flight's next frame
        s["renderer"].RenderFrame(s["cameras"][s["at"] % LOOP])
        s["at"] += 1
        return s["image"]
    if kind == "views":
        s["renderer"].RenderViews(s["cameras"])
        return s["out"]
    requests = [s["server"].submit(c, m) for c, m in s["clients"]]
    for r in requests:
        s["server"].wait(r)
    return s["out"]


def work(case):
    kind = case["kind"]
    if kind in ("sort", "scan"):
        return {"bytes": 8 * case["n"], "flops": 0}
    if kind == "unique":  # the unique values are few beside the words
        return {"bytes": 4 * case["n"], "flops": 0}
    if kind in ("views", "served"):
        pixels = sum(w * h for w, h in _sizes(case, VIEW_SIZES if kind == "views" else CLIENT_SIZES))
    else:
        pixels = case["width"] * case["height"]
    # per pixel: the image written and a hit's normal and colour read (and the
    # depth and node where they are asked for); about 120 float operations to
    # set up and shade a ray and 16 steps of about 20 through the octree
    return {"bytes": pixels * (12 + (8 if case.get("depth") else 0)), "flops": pixels * (120 + 16 * 20)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "sort":
        return torch.sort(_keys(case, seed)).values
    if kind == "scan":  # sums wrap
        return torch.cumsum(_keys(dict(case, keys="wide"), seed), 0, dtype=torch.int64).to(torch.int32)
    if kind == "unique":
        w = _words(case, seed)
        kept = w[w != NO_HIT].to(torch.int64)
        if case["nib"]:
            hits = ((torch.div((kept >> 1) - 1, case["nib"], rounding_mode="floor") + 1) << 1) | (kept & 1)
            kept = torch.where(kept > 0, hits, kept)
        u = torch.unique(kept).to(torch.int32)
        if kept.numel() < w.numel():
            u = torch.cat([u, torch.full((1,), NO_HIT, dtype=torch.int32, device=u.device)])
        out = torch.zeros_like(w)
        out[:u.numel()] = u
        return {"count": u.numel(), "unique": out}
    # images and hit nodes are whole numbers that follow from each float
    # operation's rounding, and the depth is that ray's own float sum
    return None
