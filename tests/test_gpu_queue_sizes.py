"""The work queue's kernels at batches that reach it (GRID rays and more, a remainder past it): packed rays from around the
octree, row layouts that do not divide into whole blocks, staged top levels, and the lane refill of svo_set_refill."""
import numpy as np
import pytest

import shocovox_gb300 as svo
from test_gpu_cast import assert_same_hits, both, random_rays
from test_gpu_flow import GRID, UNCOUNTED
from test_gpu_flow import random_rays as mixed_rays

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
N = GRID + 8931
W, H = 431, 331  # a camera of more than GRID rays
CAM = ([200.0, 150.0, 220.0], [64.0, 40.0, 64.0], 60.0, W, H)


@pytest.fixture(scope="module")
def scene(oracle_mod):
    return both(oracle_mod, 128, 4, svo.gen_scene(0, 128, 4, seed=91, spheres=6, octaves=2, base_freq=1.0 / 32, height_lo=4.0,
                                                  height_hi=80.0))


@pytest.fixture(scope="module")
def batches(scene):
    """label: origins, directions, the oracle's hits."""
    o, _ = scene
    rng = np.random.default_rng(7)
    odd, odd_dirs = random_rays(rng, 128, 20_000)  # axis-aligned, NaN, zero and subnormal directions among them
    few, few_dirs = mixed_rays(rng, 128, N - len(odd))
    out = {"camera": svo.gen_camera_rays(*CAM), "mixed": (np.concatenate([few, odd]), np.concatenate([few_dirs, odd_dirs]))}
    return {k: (a, d, o.cast(a, d, threads=16)) for k, (a, d) in out.items()}


@pytest.fixture
def knobs():
    lib = svo.lib()

    def turn(refill=0, depth=0, mode=0):
        for rc in (lib.svo_set_refill(refill), lib.svo_set_staging_depth(depth), lib.svo_set_cast_mode(mode)):
            svo.check(rc)

    yield turn
    turn()


def cast(p, origins, dirs, row=0, fields=tuple(svo.HIT_FIELDS)):
    n = len(origins)
    cols = {k: torch.from_numpy(np.ascontiguousarray(a[:, i])).cuda()
            for a, names in ((origins, ("ox", "oy", "oz")), (dirs, ("dx", "dy", "dz"))) for i, k in enumerate(names)}
    out = {k: torch.zeros(n + 40, dtype=getattr(torch, np.dtype(svo.HIT_FIELDS[k]).name), device="cuda") for k in fields}
    for v in out.values():
        v.fill_(0x5A)
    p.cast({k: v.data_ptr() for k, v in cols.items()}, {k: v.data_ptr() for k, v in out.items()}, n,
           torch.cuda.current_stream().cuda_stream, row)
    torch.cuda.synchronize()
    got = {k: v.cpu().numpy() for k, v in out.items()}
    assert all((v[n:] == 0x5A).all() for v in got.values()), "written past the batch"
    return {k: v[:n] for k, v in got.items()}


def check(p, batch, label, row=0, n=None):
    origins, dirs, ref = (v if isinstance(v, dict) else v[:n] for v in batch)
    ref = {k: v[:n] for k, v in ref.items()}
    assert len(origins) >= GRID
    assert_same_hits(cast(p, origins, dirs, row), ref, counters=True, label=label + ", counted")
    assert_same_hits(cast(p, origins, dirs, row, UNCOUNTED), ref, label=label)


@pytest.mark.parametrize("row", [0, W, 7, 8, 13, 64, 1000, 5000, 1 << 20])
def test_row_lengths(scene, batches, row):
    for kind in batches:
        check(scene[1], batches[kind], "%s rows %d" % (kind, row), row)
    check(scene[1], batches["camera"], "camera rows %d, partial band" % row, row, N - 37)


@pytest.mark.parametrize("depth", [1, 2, 3, 4])
def test_staging_depths(scene, batches, knobs, depth):
    knobs(depth=depth)
    check(scene[1], batches["mixed"], "staged %d" % depth)
    check(scene[1], batches["camera"], "staged %d, rows" % depth, W)


@pytest.mark.parametrize("refill", [1, 8, 21, 32])
@pytest.mark.parametrize("depth", [0, 3])
def test_refill_thresholds(scene, batches, knobs, refill, depth):
    knobs(refill, depth)
    for kind, row in (("mixed", 0), ("mixed", W), ("camera", 0), ("camera", W)):
        check(scene[1], batches[kind], "refill %d, %s, row %d" % (refill, kind, row), row)


def test_literal_form(scene, batches, knobs):
    knobs(mode=1)
    for refill in (0, 16):
        knobs(refill, mode=1)
        for kind, row in (("mixed", 0), ("camera", W)):
            check(scene[1], batches[kind], "literal, refill %d, %s" % (refill, kind), row)


def test_host_buffers(scene, batches):
    """In place (where the device can) and staged, with and without rows."""
    _, p = scene
    for mode in (0, 1, 2, 3):
        if svo.lib().svo_set_host_transfer(mode) != 0:
            continue  # the device cannot read host memory in place
        try:
            for kind, row in (("mixed", 0), ("camera", 0), ("camera", W)):
                origins, dirs, ref = batches[kind]
                label = "host mode %d, %s, row %d" % (mode, kind, row)
                assert_same_hits(p.cast_host(origins, dirs, row_length=row), ref, counters=True, label=label)
                assert_same_hits(p.cast_host(origins, dirs, fields=UNCOUNTED, row_length=row), ref, label=label)
        finally:
            svo.lib().svo_set_host_transfer(0)


def test_deep_sparse_tree(oracle_mod, knobs):
    """Eleven levels, mostly empty: restarts cross staged and unstaged levels, and the flow's node stack."""
    from helpers import COMPLEX, INSERT, ops_from
    rng = np.random.default_rng(8)
    pts = rng.integers(0, 4096, (200, 3))
    o, p = both(oracle_mod, 4096, 2, ops_from([(INSERT, int(x), int(y), int(z), COMPLEX, 0x11223344 + i, 9 + i)
                                               for i, (x, y, z) in enumerate(pts)]))
    origins, dirs = mixed_rays(rng, 4096, N)
    aimed = pts[rng.integers(0, len(pts), N // 2)] + np.float32(0.5) - origins[:N // 2]
    dirs[:N // 2] = (aimed / np.sqrt((aimed * aimed).sum(1, keepdims=True))).astype(np.float32)
    batch = (origins, dirs, o.cast(origins, dirs, threads=16))
    for refill, depth in ((0, 0), (0, 4), (1, 0), (24, 0), (32, 4)):
        knobs(refill, depth)
        check(p, batch, "deep, refill %d, depth %d" % (refill, depth))
