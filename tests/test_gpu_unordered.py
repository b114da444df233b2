"""The unordered items of a batched cast (svo_launch_config.sort_key = 1) without counters: one item is cast by
plain_kernel, several by batch_flow_kernel.  (Calls that ask for counters are cast in claim order.)"""
import numpy as np
import pytest

import shocovox_gb300 as svo
from test_gpu_cast import assert_same_hits, both
from test_gpu_cast import random_rays as special_rays
from test_gpu_flow import UNCOUNTED, random_rays

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
NOISE = dict(seed=31, occupancy=0.08, spheres=3, octaves=2, base_freq=1.0 / 16, height_lo=2.0, height_hi=24.0)


class Items:
    """Items of one call over (scene, origins, directions, row length[, the oracle's hits]); `check` compares them with the oracle."""

    def __init__(self, parts):
        self.items, self.keep = [], []
        for (o, p), origins, dirs, row, *ref in parts:
            n = len(origins)
            ref = ref[0] if ref else o.cast(origins, dirs, threads=16) if n else None
            cols = {k: torch.from_numpy(np.ascontiguousarray(a[:, i])).cuda()
                    for a, names in ((origins, ("ox", "oy", "oz")), (dirs, ("dx", "dy", "dz"))) for i, k in enumerate(names)}
            out = {k: torch.zeros(n + 33, dtype=getattr(torch, np.dtype(svo.HIT_FIELDS[k]).name), device="cuda")
                   for k in UNCOUNTED}
            self.items.append((p, {k: v.data_ptr() for k, v in cols.items()}, n, {k: v.data_ptr() for k, v in out.items()}, row))
            self.keep.append((cols, out, n, ref))

    def clear(self):
        for _, out, _, _ in self.keep:
            for v in out.values():
                v.fill_(0x5A)
        torch.cuda.synchronize()

    def check(self, label):
        torch.cuda.synchronize()
        for j, (_, out, n, ref) in enumerate(self.keep):
            got = {k: v.cpu().numpy() for k, v in out.items()}
            assert all((v[n:] == 0x5A).all() for v in got.values()), "written past item %d" % j
            if n:
                assert_same_hits({k: v[:n] for k, v in got.items()}, ref, label="%s item %d" % (label, j))

    def cast(self, ws, cfg, label):
        self.clear()
        ws.cast(self.items, cfg, torch.cuda.current_stream().cuda_stream)
        self.check(label)


def median_ms(call):
    times = []
    for _ in range(12):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        call()
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b))
    return float(np.median(times[3:]))


def spoiled(rng, dirs, share):
    """Directions of which `share` are not of unit length, so that the general forms cast them."""
    dirs = dirs.copy()
    dirs[rng.random(len(dirs)) < share] *= np.float32(1.5)
    return dirs


@pytest.mark.parametrize("share", [0.0, 0.003, 0.05, 0.5, 1.0])
@pytest.mark.parametrize("n_items", [1, 3])
def test_rays_for_the_general_forms_among_others(oracle_mod, share, n_items):
    """They wait in a warp's list until there is a warp of them, or nothing else is left, whatever their share."""
    rng = np.random.default_rng(int(share * 1000) + n_items)
    scene = both(oracle_mod, 64, 4, svo.gen_scene(3, 64, 4, **NOISE))
    parts = []
    for n in (200_003, 33, 70_001)[:n_items]:
        origins, dirs = random_rays(rng, 64, n)
        parts.append((scene, origins, spoiled(rng, dirs, share), 0))
    items, ws = Items(parts), svo.BatchWorkspace()
    for refill in (0, 1, 32):
        items.cast(ws, svo.LaunchConfig(0, 0, 0, 0, 1, 0, refill), "refill %d" % refill)
    items.cast(ws, svo.LaunchConfig(0, 0, 1, 0, 1, 0, 0), "one block per SM")


def test_directions_off_unit_length_cost_about_what_claim_order_costs(oracle_mod):
    """2^21 rays, all for the general forms: the same forms as in claim order, a warp at a time; 1.3 for two entry tests
    a ray and 6 blocks per SM instead of 7.  (Cast a claim's few at a time: 1.8.)"""
    _, p = both(oracle_mod, 256, 8, svo.gen_scene(2, 256, 8, seed=31, occupancy=0.08))
    n = 1 << 21
    origins, dirs = svo.gen_sphere_rays([128.0] * 3, 128 * np.sqrt(3.0), n, 5)
    cols = {k: torch.from_numpy(np.ascontiguousarray(a[:, i] * np.float32(f))).cuda() for a, f, names in
            ((origins, 1.0, ("ox", "oy", "oz")), (dirs, 1.5, ("dx", "dy", "dz"))) for i, k in enumerate(names)}
    status = torch.zeros(n, dtype=torch.uint8, device="cuda")
    item = [(p, {k: v.data_ptr() for k, v in cols.items()}, n, {"status": status.data_ptr()}, 0)]
    ws = svo.BatchWorkspace()

    ordered, unordered = (median_ms(lambda: ws.cast(item, svo.LaunchConfig(0, 0, 0, 0, key, 0, 0),
                                                    torch.cuda.current_stream().cuda_stream)) for key in (0, 1))
    assert unordered < 1.3 * ordered, (unordered, ordered)


@pytest.mark.parametrize("row", [0, 1920])
def test_refill_of_rays_that_keep_together_costs_about_nothing(oracle_mod, row):
    """A camera's rays are cast 32 neighbours at a time whatever svo_set_refill says; 1.3 for 6 blocks per SM instead of 7 and
    a look at the rays.  (One step of each at a time: 2.3.)"""
    _, p = both(oracle_mod, 256, 8, svo.gen_scene(1, 256, 8, seed=77, octaves=3, base_freq=1.0 / 64, height_lo=5.0,
                                                  height_hi=80.0))
    origins, dirs = svo.gen_camera_rays([40.0, 120.0, 30.0], [200.0, 20.0, 180.0], 70.0, 1920, 1080)
    n = len(origins)
    cols = {k: torch.from_numpy(np.ascontiguousarray(a[:, i])).cuda()
            for a, names in ((origins, ("ox", "oy", "oz")), (dirs, ("dx", "dy", "dz"))) for i, k in enumerate(names)}
    status = torch.zeros(n, dtype=torch.uint8, device="cuda")
    rays, hits = {k: v.data_ptr() for k, v in cols.items()}, {"status": status.data_ptr()}

    def ms(refill):
        svo.check(svo.lib().svo_set_refill(refill))
        try:
            return median_ms(lambda: p.cast(rays, hits, n, torch.cuda.current_stream().cuda_stream, row))
        finally:
            svo.lib().svo_set_refill(0)

    off, on = ms(0), ms(24)
    assert on < 1.3 * off, (on, off)


def odd_items(oracle_mod, seed):
    """Scenes of several sizes and brick dimensions, with empty and 1-ray items, a remainder, and items in claim order."""
    rng = np.random.default_rng(seed)
    parts = []
    for j, (kind, size, dim, n, row) in enumerate([(0, 128, 4, 6000, 0), (3, 64, 2, 1, 0), (3, 32, 8, 0, 0), (1, 64, 8, 33, 0),
                                                   (2, 256, 8, 20000, 0), (3, 64, 1, 2500, 40), (0, 64, 4, 3000, 0),
                                                   (3, 64, 4, 0, 0), (3, 64, 4, 3200, 64), (3, 32, 8, 0, 0)]):
        scene = both(oracle_mod, size, dim, svo.gen_scene(kind, size, dim, seed=seed + j, occupancy=0.1, spheres=3, octaves=2,
                                                          base_freq=1.0 / 16, height_lo=2.0, height_hi=size * 0.4))
        origins, dirs = special_rays(rng, size, n)
        parts.append((scene, origins, dirs, row, scene[0].cast(origins, dirs, threads=16) if n else None))
    return parts


@pytest.fixture
def cast_mode():
    yield lambda mode: svo.check(svo.lib().svo_set_cast_mode(mode))
    svo.lib().svo_set_cast_mode(0)


def test_several_items(oracle_mod, cast_mode):
    """Launch configurations, both cast modes, one call after another on a workspace; an item alone; no unordered item at all."""
    parts = odd_items(oracle_mod, 700)
    ws = svo.BatchWorkspace()
    for mode in (0, 1):
        cast_mode(mode)
        items = Items(parts)
        configs = ((0, 0, 0, 0, 1, 0, 0), (64, 32, 0, 0, 1, 2, 1), (128, 100, 0, 4, 1, 0, 8), (96, 256, 3, 0, 1, 4, 32),
                   (32, 64, 1, 5, 1, 0, 24))
        for cfg in configs if mode == 0 else configs[:2]:  # rays that reach the work cap take a second a call
            items.cast(ws, svo.LaunchConfig(*cfg), "mode %d, %s" % (mode, cfg))
        for only in ([4], [1], [2, 3], [5, 8], [2, 7, 9], [6, 0]) if mode == 0 else ([1], [2, 3]):
            Items([parts[k] for k in only]).cast(ws, svo.LaunchConfig(0, 0, 0, 0, 1, 0, 0), "mode %d, items %s" % (mode, only))


def test_workspace_grows_between_calls_and_before_a_graph(oracle_mod):
    parts = odd_items(oracle_mod, 900)
    small, large = Items(parts[:1]), Items((parts * 3)[:25])
    ws, cfg = svo.BatchWorkspace(), svo.LaunchConfig(0, 0, 0, 0, 1, 0, 0)
    for items, label in ((small, "small"), (large, "grown"), (small, "small again")):
        items.cast(ws, cfg, label)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        ws.cast(large.items, cfg, stream.cuda_stream)
    for k in range(3):
        large.clear()
        graph.replay()
        large.check("replay %d" % k)


@pytest.mark.parametrize("n", [1, 8, 9, 31, 32, 33, 40, 41, 127, 129, 131071, 131072])
def test_sizes_of_a_lone_item(oracle_mod, n):
    scene = both(oracle_mod, 64, 4, svo.gen_scene(3, 64, 4, **NOISE))
    ws = svo.BatchWorkspace()
    camera = tuple(a[:n] for a in svo.gen_camera_rays([150.0, 90.0, 140.0], [32.0, 16.0, 32.0], 50.0, 431, 331))
    for label, (origins, dirs) in (("random", random_rays(np.random.default_rng(n), 64, n)), ("camera", camera)):
        Items([(scene, origins, dirs, 0)]).cast(ws, svo.LaunchConfig(0, 0, 0, 0, 1, 0, 0), "%s %d" % (label, n))
