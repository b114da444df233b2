"""Host-buffer casts over arrays that the device cannot use in place (svo_cast_host reads and writes small batches and
camera rows where they lie): the hits have to be those of the same call over arrays of its own."""

import numpy as np
import pytest

import shocovox_gb300 as svo
from shocovox_gb300._lib import SvoError
from test_gpu_cast import assert_same_hits, both
from test_gpu_flow import random_rays

pytestmark = pytest.mark.gpu
NAMES = ("ox", "oy", "oz", "dx", "dy", "dz")


@pytest.fixture(scope="module")
def scene(oracle_mod):
    return both(oracle_mod, 64, 4, svo.gen_scene(3, 64, 4, seed=8, occupancy=0.1, spheres=2))


def shifted(a, off):
    """A copy of `a` whose first byte lies `off` bytes past a 16-byte boundary."""
    raw = np.empty(a.nbytes + 64, np.uint8)
    at = (-raw.ctypes.data) % 16 + off
    out = raw[at:at + a.nbytes].view(a.dtype)
    out[...] = a
    return out


@pytest.mark.parametrize("n,row", [(1, 0), (33, 0), (20000, 0), (20000, 200), (431 * 331, 431)])
@pytest.mark.parametrize("off", [1, 2, 3])
def test_arrays_off_their_alignment(scene, n, row, off):
    o, p = scene
    origins, dirs = random_rays(np.random.default_rng(n + off), 64, n)
    ref = o.cast(origins, dirs, threads=16)
    cols = [np.ascontiguousarray(a[:, k]) for a in (origins, dirs) for k in range(3)]
    plain = {k: np.zeros(n, t) for k, t in svo.HIT_FIELDS.items()}
    for which in ("rays", "hits", "one field"):
        ins = [shifted(c, off if which == "rays" else 0) for c in cols]
        out = {k: shifted(v, off if which == "hits" or (which == "one field" and k == "albedo") else 0)
               for k, v in plain.items()}
        p.cast_host_soa(ins, out, 0, row)
        assert_same_hits(out, ref, counters=True, label="%s off by %d" % (which, off))


def test_in_place_access_of_unaligned_arrays_is_refused(scene):
    _, p = scene
    origins, dirs = random_rays(np.random.default_rng(1), 64, 100)
    cols = [shifted(np.ascontiguousarray(a[:, k]), 1) for a in (origins, dirs) for k in range(3)]
    out = {"status": np.zeros(100, np.uint8)}
    svo.check(svo.lib().svo_set_host_transfer(2))
    try:
        with pytest.raises(SvoError):
            p.cast_host_soa(cols, out)
    finally:
        svo.check(svo.lib().svo_set_host_transfer(0))


@pytest.mark.parametrize("n", [2, 1000, 20000])
@pytest.mark.parametrize("field,off", [("status", 0), ("brick_octant", 1), ("px", 0), ("px", 4), ("albedo", -4), ("nz", 400),
                                       ("entry_kind", -1)])
def test_hits_over_the_rays(scene, n, field, off):
    """A field that lies over a ray array, element for element or not."""
    o, p = scene
    origins, dirs = random_rays(np.random.default_rng(n), 64, n)
    ref = o.cast(origins, dirs, threads=16)
    raw = np.zeros(6 * 4 * n + 4096, np.uint8)  # the six ray arrays, one after the other
    base = (-raw.ctypes.data) % 16 + 1024
    cols = [raw[base + 4 * n * k:base + 4 * n * (k + 1)].view(np.float32) for k in range(6)]
    for k, c in enumerate(cols):
        c[...] = origins[:, k] if k < 3 else dirs[:, k - 3]
    at = base + 4 * n * 1 + off  # over oy
    out = {k: np.zeros(n, t) for k, t in svo.HIT_FIELDS.items() if k != field}
    kind = np.dtype(svo.HIT_FIELDS[field])
    out[field] = raw[at:at + kind.itemsize * n].view(kind)
    p.cast_host_soa(cols, out)
    assert_same_hits(out, ref, counters=True, label="%s at %d" % (field, off))
