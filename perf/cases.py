"""The ray-cast work that users of the framework have it do, as cases for a timing harness.

A case names an entry point (`api`), a scene recipe and the sizes of one call.  `prepare` gives what a
program holds before the call (an uploaded scene, rays in device or host memory, output buffers),
`run` makes the call, `work` counts what it cannot do without and `exact` computes the impact points
in 64 bits by marching a dense voxel grid, independent of the framework.
"""
import ctypes
import math

import numpy as np
import torch

import shocovox_gb300 as svo

RAY = ("ox", "oy", "oz", "dx", "dy", "dz")
POINT, NORMAL = ("px", "py", "pz"), ("nx", "ny", "nz")
COUNTERS = ("node_visits", "child_reads", "voxel_reads", "run_visits")
ALL = tuple(k for k in svo.HIT_FIELDS if k not in COUNTERS)
# what a renderer reads of a hit
SHADE = ("status", "entry_kind", "albedo", "user") + POINT + NORMAL

# Scene recipes by name (seeded, built once in a process and kept like any loaded scene).
SCENES = {
    # value-noise heightfields with solid spheres
    "height64": dict(kind=0, size=64, brick_dim=4, seed=42, spheres=4, octaves=2, base_freq=1.0 / 16, height_lo=2.0,
                     height_hi=24.0),
    "height128": dict(kind=0, size=128, brick_dim=4, seed=0x5EED0001, spheres=32, octaves=2, base_freq=1.0 / 32,
                      height_lo=0.0, height_hi=96.0),
    # terrain with caves
    "terrain256": dict(kind=1, size=256, brick_dim=8, seed=0x5EED0002, octaves=3, base_freq=1.0 / 64, height_lo=5.12,
                       height_hi=84.48, cave_threshold=0.55),
    "terrain512": dict(kind=1, size=512, brick_dim=8, seed=0x5EED0002, octaves=3, base_freq=1.0 / 128,
                       height_lo=10.24, height_hi=168.96, cave_threshold=0.55),
    # sparse solid and noise-carved blocks
    "sparse512": dict(kind=2, size=512, brick_dim=8, seed=0x5EED0003, occupancy=0.05),
    # boxes of large cells
    "boxes1024": dict(kind=4, size=1024, brick_dim=8, seed=0x5EED0005, occupancy=0.03),
    "boxes256": dict(kind=4, size=256, brick_dim=8, seed=0x5EED0024, occupancy=0.02),
}
# 3D noise with spheres at every brick dimension in use
for _k, (_s, _d, _o) in enumerate([(64, 2, 0.05), (64, 4, 0.2), (64, 8, 0.1), (128, 2, 0.08), (128, 4, 0.02),
                                   (128, 8, 0.15), (256, 4, 0.03), (256, 8, 0.06)]):
    SCENES["noise%d_%d" % (_s, _d)] = dict(kind=3, size=_s, brick_dim=_d, seed=0x5EED0004 + 17 * _k, occupancy=_o,
                                           spheres=8, octaves=2, base_freq=1.0 / 32)
NOISE = tuple(k for k in SCENES if k.startswith("noise"))
SERVED = ("boxes1024", "boxes256", "terrain256", "noise128_8")
RESOLUTIONS = ((320, 240), (640, 480), (1280, 720), (1920, 1080))


def listed():
    return [
        # picking: the voxel under the mouse, one ray in host memory, every field back
        dict(name="pick_one", api="host", scene="height64", n=1),
        # a game's line-of-sight probes of one frame, on the device
        dict(name="probes_1000", api="cast", scene="height128", rays="random", n=1000, fields="all", refill=0),
        # a small preview image
        dict(name="image_640x480", api="rows", scene="height128", width=640, height=480, cams=1, fields="shade"),
        # the headline: four full-HD cameras over 512^3 terrain
        dict(name="terrain_4x1080p", api="rows", scene="terrain512", width=1920, height=1080, cams=4, fields="shade"),
        # an odd-sized image whose caller gives no row length
        dict(name="image_plain_1283x721", api="cast", scene="terrain256", rays="camera", n=1283 * 721, width=1283,
             fields="all", refill=0),
        # rays in no order (light transport, sensor simulation)
        dict(name="incoherent_4M", api="cast", scene="sparse512", rays="random", n=1 << 22, fields="shade", refill=0),
        # the same kind of rays through the batched cast's ray sort with lane refill
        dict(name="sorted_1M", api="batch", scene="sparse512", items=1, n=(1 << 20) + 13, sort=1, refill=24),
        # many small scenes in one launch: half of each batch camera rows, half random rays
        dict(name="multiscene_24", api="batch", scene="noise", items=24, n=200000, sort=0, refill=0),
        # level of detail through MIP maps
        dict(name="lod_1080p", api="lod", scene="terrain256", width=1920, height=1080, distance=256.0),
        # the example's frame: rays, cast and shading in one call, four views
        dict(name="render_4x1080p", api="render", scene="terrain512", width=1920, height=1080, views=4),
        # a full-HD camera whose rays and hits live in pinned host memory
        dict(name="host_1080p", api="host_rows", scene="terrain256", width=1920, height=1080),
        # a burst of camera requests to the server
        dict(name="serve_24", api="serve", requests=24),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    api = rng.choice(["host", "cast", "cast", "rows", "rows", "batch", "batch", "lod", "render", "host_rows", "serve"])
    small = ["height64", "height128", "terrain256", "sparse512", "boxes1024"] + list(NOISE)
    width, height = _log(rng, 33, 1920), _log(rng, 17, 1080)
    if api == "host":
        return dict(api=api, scene=rng.choice(small), n=_log(rng, 1, 20000))
    if api == "cast":
        rays = rng.choice(["random", "camera"])
        return dict(api=api, scene=rng.choice(small), rays=rays, n=_log(rng, 40, 1 << 22), width=width,
                    fields=rng.choice(["all", "shade"]), refill=rng.choice([0, 0, 16, 24]) if rays == "random" else 0)
    if api == "rows":
        return dict(api=api, scene=rng.choice(small), width=width, height=height, cams=rng.randint(1, 3),
                    fields=rng.choice(["all", "shade"]))
    if api == "batch":
        if rng.random() < 0.5:
            return dict(api=api, scene="sparse512", items=rng.randint(1, 3), n=_log(rng, 2000, 1 << 20), sort=1,
                        refill=rng.choice([0, 16, 24, 32]))
        return dict(api=api, scene="noise", items=rng.randint(2, 24), n=_log(rng, 2000, 200000), sort=0, refill=0)
    if api == "lod":
        return dict(api=api, scene="terrain256", width=width, height=height,
                    distance=float(_log(rng, 16, 1024)))
    if api == "render":
        return dict(api=api, scene=rng.choice(small), width=width, height=height,
                    views=min(rng.randint(1, 18), max(1, 4 * 1920 * 1080 // (width * height))))
    if api == "host_rows":
        return dict(api=api, scene=rng.choice(small), width=width, height=height)
    return dict(api=api, requests=rng.randint(1, 24))


# ---- scenes ----------------------------------------------------------------------------------------
_scenes = {}


def _ops(name):
    r = dict(SCENES[name])
    return svo.gen_scene(r.pop("kind"), r.pop("size"), r.pop("brick_dim"), r.pop("seed"), **r)


def _scene(name, mips=False):
    """The uploaded scene of a recipe."""
    if (name, mips) not in _scenes:
        t = svo.Octree(SCENES[name]["size"], SCENES[name]["brick_dim"])
        t.apply_ops(_ops(name))
        if mips:
            t.switch_albedo_mip_maps(True)
        t.upload(_stream())
        torch.cuda.synchronize()
        _scenes[name, mips] = t
    return _scenes[name, mips]


def _stream():
    return torch.cuda.current_stream().cuda_stream


# ---- rays ------------------------------------------------------------------------------------------
def _unit(v):
    return v / torch.sqrt((v * v).sum(1, keepdim=True))


def _camera_pose(rng, name):
    """Over the terrain, looking down at it, or outside the other scenes, looking at their middle."""
    S = float(SCENES[name]["size"])
    if name.startswith("terrain"):
        return ([rng.uniform(0.15, 0.85) * S, 0.45 * S, rng.uniform(0.15, 0.85) * S],
                [rng.uniform(0.1, 0.9) * S, 0.1 * S, rng.uniform(0.1, 0.9) * S], 70.0)
    a, el = rng.uniform(0, 2 * np.pi), rng.uniform(0.35, 0.7)
    eye = [S / 2 + 1.5 * S * np.cos(el) * np.cos(a), S / 2 + 1.5 * S * np.sin(el), S / 2 + 1.5 * S * np.cos(el) * np.sin(a)]
    return eye, [S / 2 + rng.uniform(-0.1, 0.1) * S, S / 2, S / 2 + rng.uniform(-0.1, 0.1) * S], 60.0


def _camera(rng, name, width, height):
    """A pinhole camera's rays in raster order: (n, 3) origins and directions."""
    eye, target, fov = _camera_pose(rng, name)
    dev = torch.device("cuda")
    e, t = (torch.tensor(v, dtype=torch.float32, device=dev) for v in (eye, target))
    fwd = _unit((t - e)[None])[0]
    up = torch.tensor([0.0, 1.0, 0.0], device=dev)
    right = _unit(torch.linalg.cross(up, fwd)[None])[0]
    tan = math.tan(math.radians(fov) / 2)
    u = (2 * (torch.arange(width, device=dev) + 0.5) / width - 1) * (tan * width / height)
    v = (1 - 2 * (torch.arange(height, device=dev) + 0.5) / height) * tan
    d = (fwd + right * u[None, :, None] + up * v[:, None, None]).reshape(-1, 3)
    return e.expand(d.shape[0], 3), _unit(d)


def _random(seed, name, n):
    """Origins on the scene's bounding sphere, directions in no order."""
    S = float(SCENES[name]["size"])
    g = torch.Generator(device="cuda").manual_seed(seed)
    o = _unit(torch.randn((n, 3), generator=g, device="cuda")) * (S * math.sqrt(3) / 2) + S / 2
    return o, _unit(torch.randn((n, 3), generator=g, device="cuda"))


def _item_rays(case, k):
    """Rays of item k of a batch over many scenes: 1,000 to n, spread over the logarithm."""
    return int(1000 * (case["n"] / 1000) ** ((k * 0.6180339887) % 1))


def _rays_of(case, seed):
    """[(scene name, origins, directions, row length)] of a cast case."""
    rng = np.random.default_rng(seed)
    api = case["api"]
    if api == "batch":
        out = []
        for k in range(case["items"]):
            if case["sort"]:
                out.append((case["scene"],) + _random(seed * 1000 + k, case["scene"], case["n"] - 7 * k) + (0,))
                continue
            name = NOISE[k % len(NOISE)]
            n = _item_rays(case, k)
            if k % 2:
                out.append((name,) + _random(seed * 1000 + k, name, n) + (0,))
            else:
                w = max(1, int(math.sqrt(n * 16 / 9)))
                out.append((name,) + _camera(rng, name, w, max(1, n // w)) + (w,))
        return out
    name = case["scene"]
    if api == "host":  # picking from a camera outside, or probes
        o, d = _camera(rng, name, 31, 31) if case["n"] == 1 else _random(seed, name, case["n"])
        k = 480 if case["n"] == 1 else 0
        return [(name, o[k:k + case["n"]], d[k:k + case["n"]], 0)]
    if api == "cast" and case["rays"] == "random":
        return [(name,) + _random(seed, name, case["n"]) + (0,)]
    if api == "cast":
        o, d = _camera(rng, name, case["width"], -(-case["n"] // case["width"]))
        return [(name, o[:case["n"]], d[:case["n"]], 0)]
    cams = [_camera(rng, name, case["width"], case["height"]) for _ in range(case.get("cams", 1))]
    return [(name, torch.cat([o for o, _ in cams]), torch.cat([d for _, d in cams]), case["width"])]


def _soa(o, d):
    return {k: c.contiguous() for k, c in zip(RAY, list(o.unbind(1)) + list(d.unbind(1)))}


def _outputs(n, fields):
    kinds = {np.dtype(np.uint8): torch.uint8, np.dtype(np.uint32): torch.int32, np.dtype(np.float32): torch.float32}
    return {k: torch.empty(n, dtype=kinds[np.dtype(svo.HIT_FIELDS[k])], device="cuda") for k in fields}


def _ptrs(tensors):
    return {k: t.data_ptr() for k, t in tensors.items()}


# ---- one case --------------------------------------------------------------------------------------
def prepare(case, seed):
    api = case["api"]
    s = dict(api=api, case=case)
    if api == "serve":
        rng = np.random.default_rng(seed)
        s["server"] = svo.Server()
        ids = {name: s["server"].add_scene(_scene(name)) for name in SERVED}
        s["requests"] = []
        for k in range(case["requests"]):
            name = SERVED[int(rng.integers(len(SERVED)))]
            w, h = RESOLUTIONS[k % len(RESOLUTIONS)]
            out = {"status": np.empty(w * h, np.uint8), "albedo": np.empty(w * h, np.uint32)}
            s["requests"].append((ids[name],) + _camera_pose(rng, name) + (w, h, out))
        return s
    if api == "render":
        rng = np.random.default_rng(seed)
        s["scene"] = _scene(case["scene"])
        S = float(SCENES[case["scene"]]["size"])
        s["views"] = []
        for _ in range(case["views"]):
            v = svo.orbit_viewport(rng.uniform(0, 2 * np.pi), 1.1 * S)
            o = np.array(list(v.origin), np.float32) + np.float32(S / 2)
            d = np.array([S / 2, 0.2 * S, S / 2], np.float32) - o
            d = d / np.sqrt((d[0] * d[0] + d[1] * d[1]) + d[2] * d[2], dtype=np.float32)
            s["views"].append(svo.viewport(o, d, fov=2.0))
        s["rgba"] = torch.empty((case["views"], case["height"], case["width"], 4), dtype=torch.uint8, device="cuda")
        return s
    sets = _rays_of(case, seed)
    if api == "batch":
        s["workspace"] = svo.BatchWorkspace()
        s["config"] = svo.LaunchConfig(0, 0, 0, 0, case["sort"], 0, case["refill"])
        s["rays"] = [_soa(o, d) for _, o, d, _ in sets]
        # one array per field for the whole batch, an item's hits in its slice
        ends = np.cumsum([len(o) for _, o, _, _ in sets])
        s["out"] = _outputs(int(ends[-1]), SHADE)
        s["items"] = [(_scene(name), _ptrs(r), len(o), _ptrs({k: t[end - len(o):end] for k, t in s["out"].items()}), row)
                      for (name, o, _, row), r, end in zip(sets, s["rays"], ends)]
        return s
    name, o, d, row = sets[0]
    s["scene"], s["n"], s["row"] = _scene(name, api == "lod"), len(o), row
    if api == "host":
        s["o"], s["d"] = o.cpu().numpy(), d.cpu().numpy()
        return s
    s["rays"] = _soa(o, d)
    fields = ALL if case.get("fields") == "all" else SHADE
    if api == "host_rows":
        s["rays"] = {k: t.cpu().pin_memory() for k, t in s["rays"].items()}
        s["cols"] = [s["rays"][k].numpy() for k in RAY]
        s["out"] = {k: torch.empty(t.shape, dtype=t.dtype).pin_memory() for k, t in _outputs(s["n"], fields).items()}
        s["arrays"] = {k: t.numpy() for k, t in s["out"].items()}
        return s
    s["out"] = _outputs(s["n"], fields)
    s["rp"], s["hp"] = _ptrs(s["rays"]), _ptrs(s["out"])
    return s


def run(s):
    api, case = s["api"], s["case"]
    if api == "host":
        return s["scene"].cast_host(s["o"], s["d"], fields=ALL)
    if api == "host_rows":
        s["scene"].cast_host_soa(s["cols"], s["arrays"], _stream(), s["row"])
        return s["out"]
    if api == "serve":
        ids = [s["server"].submit(*r) for r in s["requests"]]
        for i in ids:
            s["server"].wait(i)
        return [r[-1] for r in s["requests"]]
    if api == "render":
        s["scene"].render_viewports(s["views"], case["width"], case["height"], s["rgba"].data_ptr(), 0, _stream())
        return s["rgba"]
    if api == "batch":
        s["workspace"].cast(s["items"], s["config"], _stream())
        return s["out"]
    if api == "lod":
        s["scene"].cast_lod(s["rp"], s["hp"], s["n"], case["distance"], _stream(), s["row"])
        return s["out"]
    if case.get("refill"):
        svo.lib().svo_set_refill(ctypes.c_int32(case["refill"]))
    s["scene"].cast(s["rp"], s["hp"], s["n"], _stream(), s["row"])
    if case.get("refill"):
        svo.lib().svo_set_refill(ctypes.c_int32(0))
    return s["out"]


def _hit_bytes(fields):
    return sum(np.dtype(svo.HIT_FIELDS[k]).itemsize for k in fields)


def work(case):
    """Rays in and hit fields out (the scene's part that rays read is the traversal's own), and the
    operations of one slab test and one impact per ray."""
    api = case["api"]
    if api == "serve":
        n = sum(w * h for w, h in (RESOLUTIONS[k % len(RESOLUTIONS)] for k in range(case["requests"])))
        per = 5
    elif api == "render":
        n, per = case["views"] * case["width"] * case["height"], 4
    elif api == "batch":
        n = sum(case["n"] if case["sort"] else _item_rays(case, k) for k in range(case["items"]))
        per = 24 + _hit_bytes(SHADE)
    elif api in ("cast", "host"):
        n, per = case["n"], 24 + _hit_bytes(ALL if api == "host" or case["fields"] == "all" else SHADE)
    else:
        n = case["width"] * case["height"] * case.get("cams", 1)
        per = 24 + _hit_bytes(ALL if case.get("fields") == "all" else SHADE)
    return {"bytes": float(n * per), "flops": float(n * 100)}


# ---- the same impacts in 64 bits -------------------------------------------------------------------
_grids = {}


def _grid(name):
    """The scene's voxels as a dense boolean grid, from its recipe's operations."""
    if name not in _grids:
        ops, S = _ops(name), SCENES[name]["size"]
        g = np.zeros((S, S, S), bool)
        one = ops["size"] <= 1
        g[ops["x"][one], ops["y"][one], ops["z"][one]] = True
        for x, y, z, k in zip(*(ops[f][~one].tolist() for f in ("x", "y", "z", "size"))):
            g[x:x + k, y:y + k, z:z + k] = True
        _grids.clear()
        _grids[name] = torch.from_numpy(g).cuda().reshape(-1)
    return _grids[name]


def _march(name, o, d):
    """First impact points of rays on the grid: (n, 3), zero where a ray hits nothing."""
    grid, S = _grid(name), SCENES[name]["size"]
    point = torch.zeros((len(o), 3), dtype=torch.float64, device="cuda")
    d = torch.where(d == 0, torch.full_like(d, 1e-300), d)
    near, far = torch.minimum(-o / d, (S - o) / d), torch.maximum(-o / d, (S - o) / d)
    t = near.max(1)[0].clamp(min=0)
    at = torch.nonzero((far.min(1)[0] >= t)).flatten()
    o, d, t = o[at], d[at], t[at]
    cell = (o + d * t[:, None]).floor().clamp(0, S - 1)
    nxt, delta, step = (cell + (d > 0) - o) / d, 1 / d.abs(), torch.sign(d).long()
    cell = cell.long()
    for _ in range(3 * S + 3):
        if not len(at):
            break
        hit = grid[(cell[:, 0] * S + cell[:, 1]) * S + cell[:, 2]]
        h = torch.nonzero(hit).flatten()
        if len(h):
            point[at[h]] = o[h] + d[h] * t[h, None]
        t, axis = nxt.min(1)
        one = torch.zeros_like(step).scatter_(1, axis[:, None], 1)
        cell = cell + step * one
        nxt = nxt + delta * one
        stay = torch.nonzero(~hit & ((cell >= 0) & (cell < S)).all(1)).flatten()
        if len(stay) < len(at):
            at, o, d, t, cell, nxt, delta, step = (v[stay] for v in (at, o, d, t, cell, nxt, delta, step))
    return point


def exact(case, seed):
    """The impact points.  Normals have no such value: an impact on a voxel's edge has a diagonal one,
    and which impacts lie on an edge is decided by the last bits of the point in 32 bits."""
    if case["api"] in ("serve", "render", "lod"):  # bytes; a MIP's own geometry
        return None
    points = []
    for name, o, d, _ in _rays_of(case, seed):
        points += [_march(name, o[k:k + (1 << 21)].double(), d[k:k + (1 << 21)].double()) for k in range(0, len(o), 1 << 21)]
    got = {k: None for k in (ALL if case["api"] == "host" or case.get("fields") == "all" else SHADE)}
    got.update((k, c.contiguous()) for k, c in zip(POINT, torch.cat(points).unbind(1)))
    return got
