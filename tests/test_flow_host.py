"""The unit-direction form of the cast (shocovox_gb300/csrc/svo_flow.cuh), compiled for the host, against the
oracle: every record bit for bit over the rays it accepts, on scenes of every brick dimension and deep
trees, with rays along axes and diagonals, from grid points, and nearly parallel to the cell planes.
Rays it leaves to the general forms (directions that are not unit, far origins) are only counted."""
import ctypes
import glob
import os
import shutil
import subprocess

import numpy as np
import pytest

import shocovox_gb300 as svo
from helpers import COMPLEX, INSERT, ops_from

HERE = os.path.dirname(os.path.abspath(__file__))
LIB = os.path.join(os.path.dirname(HERE), "shocovox_gb300", "_lib")
N = 4000


@pytest.fixture(scope="module")
def flow(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("needs nvcc")
    so = str(tmp_path_factory.mktemp("flow") / "flow_check.so")
    objects = [o for o in glob.glob(os.path.join(LIB, "*.o")) if not o.endswith("svo_device.o")]
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O1", "-std=c++17", "-fmad=false", "-Xcompiler",
                    "-fPIC,-O2,-ffp-contract=off,-frounding-math", "-shared", os.path.join(HERE, "flow_check.cu")] + objects +
                   ["-o", so, "-lpthread", "-ldl"], check=True, capture_output=True)
    return ctypes.CDLL(so)


def unit(v):
    v = np.asarray(v, np.float32)
    return v / np.sqrt((v * v).sum(1, keepdims=True), dtype=np.float32)


def rays(rng, S, kind):
    o, d = rng.uniform(-0.2 * S, 1.2 * S, (N, 3)), rng.normal(size=(N, 3))
    if kind == "grid":
        o, d = rng.integers(0, S + 1, (N, 3)), rng.integers(-3, 4, (N, 3)) + np.array([0, 0, 1e-9])
    elif kind == "axis":
        d = np.zeros((N, 3))
        d[np.arange(N), rng.integers(0, 3, N)] = rng.choice([-1, 1], N)
    elif kind == "diagonal":
        o, d = rng.integers(-2, S + 3, (N, 3)), rng.choice([-1, 1], (N, 3))
    elif kind == "grazing":
        d[np.arange(N), rng.integers(0, 3, N)] *= 10.0 ** -rng.uniform(2, 9, N)
    return np.ascontiguousarray(o, np.float32), np.ascontiguousarray(unit(d))


def scene(name, rng):
    g = svo.gen_scene
    if name.startswith("deep"):
        S, D = (4096, 2) if name == "deep4096" else (2048, 1)
        pts = rng.integers(0, S, (200, 3))
        return S, D, ops_from([(INSERT, int(x), int(y), int(z), COMPLEX, 0xAABBCCFF, i + 1)
                               for i, (x, y, z) in enumerate(pts)]), pts
    S, D = {"height": (64, 4), "dim1": (32, 1), "dim2": (64, 2), "dim8": (64, 8), "dim16": (64, 16), "boxes": (256, 8),
            "sparse": (128, 8)}[name]
    kind = {"height": 0, "boxes": 4, "sparse": 2}.get(name, 3)
    return S, D, g(kind, S, D, 11, occupancy=0.05 if kind != 3 else 0.1, spheres=3, octaves=2, base_freq=1.0 / 16,
                   height_lo=2.0, height_hi=S * 0.4), None


@pytest.mark.parametrize("name", ["height", "dim1", "dim2", "dim8", "dim16", "boxes", "sparse", "deep4096", "deep2048"])
def test_unit_form_matches_the_oracle(flow, oracle_mod, name):
    rng = np.random.default_rng(len(name) * 7 + 1)
    S, D, ops, pts = scene(name, rng)
    h = ctypes.c_void_p()
    assert flow.svo_scene_create(S, D, ctypes.byref(h)) == 0
    ops = np.ascontiguousarray(ops, dtype=svo.OP_DTYPE)
    done = ctypes.c_uint64()
    vp = lambda a: ctypes.c_void_p(a.ctypes.data)  # noqa: E731
    assert flow.svo_apply_ops(h, vp(ops), ctypes.c_uint64(len(ops)), ctypes.byref(done)) == 0
    tree = oracle_mod.Tree(S, D)
    tree.apply_ops(ops)
    for kind in ("random", "grid", "axis", "diagonal", "grazing"):
        o, d = rays(rng, S, kind)
        if pts is not None:  # half of them at the few voxels of a deep tree
            d[:N // 2] = unit(pts[rng.integers(0, len(pts), N // 2)] + np.float32(0.5) - o[:N // 2])
        form, rec = np.zeros(N, np.uint8), np.zeros((N, 12), np.uint32)
        flow.flow_check(h, vp(o), vp(d), ctypes.c_uint64(N), vp(form), vp(rec))
        ref = tree.cast(o, d, threads=8)
        exp = np.zeros((N, 12), np.uint32)
        exp[:, 0] = ref["status"]
        for k, f in enumerate(("brick_octant", "node_key", "voxel_index", "pix")):
            exp[:, 1 + k] = ref[f]
        for k, f in enumerate(("px", "py", "pz", "nx", "ny", "nz")):
            exp[:, 5 + k] = (ref[f] + np.float32(0)).view(np.uint32)  # -0 as 0
        exp[ref["status"] != 1, 1:] = 0
        rec[:, 5:11] = (rec[:, 5:11].view(np.float32) + np.float32(0)).view(np.uint32)
        cast = form == 1
        assert cast.sum() > N // 2, kind
        bad = np.nonzero((rec != exp).any(1) & cast)[0]
        assert len(bad) == 0, "%s rays, ray %d: %s, expected %s" % (kind, bad[0], rec[bad[0]], exp[bad[0]])
    flow.svo_scene_destroy(h)


def test_rays_left_to_the_general_forms(flow, oracle_mod):
    h = ctypes.c_void_p()
    assert flow.svo_scene_create(64, 4, ctypes.byref(h)) == 0
    far = np.float32(64 * 1024)
    cases = [((1, 1, 1), (0, 0, 1), 1), ((1, 1, 1), (0, 0, 2), 0), ((1, 1, 1), (0, 0, 0), 0), ((1, 1, 1), (np.nan, 0, 1), 0),
             ((np.inf, 1, 1), (0, 0, 1), 0), ((far, 1, 1), (-1, 0, 0), 1), ((far * 2, 1, 1), (-1, 0, 0), 0),
             ((1, 1, 1), (-0.0, 0, 1), 0), ((1, 1, 1), (np.float32(-1e-9), 0, 1), 0)]
    o = np.array([c[0] for c in cases], np.float32)
    d = np.array([c[1] for c in cases], np.float32)
    form, rec = np.zeros(len(o), np.uint8), np.zeros((len(o), 12), np.uint32)
    vp = lambda a: ctypes.c_void_p(a.ctypes.data)  # noqa: E731
    flow.flow_check(h, vp(o), vp(d), ctypes.c_uint64(len(o)), vp(form), vp(rec))
    assert [int(v != 0) for v in form] == [c[2] for c in cases]
    flow.svo_scene_destroy(h)


@pytest.mark.parametrize("width", [96, 127, 240, 320, 640, 960, 1024, 1280, 1283, 1920, 2048, 2560, 3840, 4096])
def test_sampled_pairs_of_an_image_stay_in_their_rows(flow, width):
    """At most 8 of the 32 pairs may straddle a row's end, or a camera's rays would be cast as rays in no order."""
    flow.flow_pair.restype, flow.flow_pair.argtypes = ctypes.c_uint64, [ctypes.c_uint64, ctypes.c_uint32]
    apart = flow.flow_pair_apart()
    for ratio in (9 / 16, 3 / 4, 1):
        rows = int(width * ratio)
        for images in range(1, 33):
            n = width * rows * images
            if n < 1 << 19:
                continue
            at = [flow.flow_pair(n, k) for k in range(32)]
            assert all(a < b for a, b in zip(at, at[1:])) and at[-1] + apart < n
            assert sum(a % width + apart >= width for a in at) <= 8, (width, rows, images)
    for n in (1, 8, 9, 31, 40, 41, 64, 1 << 19, 1 << 33):
        assert all(flow.flow_pair(n, k) + (apart if n > apart else 0) < n for k in range(32)), n
