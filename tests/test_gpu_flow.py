"""GPU parity of large batches without a row layout (plain_kernel): rays in no order, which the warps hand to
idle lanes one by one, and cameras in raster order; rays that the unit form does not take among them; the
sizes at which a batch changes kernels; casts one after another on a stream share its work counter."""
import numpy as np
import pytest

import shocovox_gb300 as svo
from test_gpu_cast import assert_same_hits, both

pytestmark = pytest.mark.gpu
UNCOUNTED = tuple(k for k in svo.HIT_FIELDS if k not in ("node_visits", "child_reads", "voxel_reads", "run_visits"))
GRID, FLOW = 1 << 17, 1 << 19  # kQueueMinRays, kFlowMinRays


def random_rays(rng, S, n):
    o = rng.uniform(-0.3 * S, 1.3 * S, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    return o, d / np.sqrt((d * d).sum(1, keepdims=True), dtype=np.float32)


def device_cast(p, origins, dirs, casts=1):
    """The uncounted fields of a device cast; checks that nothing is written past the batch."""
    torch = pytest.importorskip("torch")
    n = len(origins)
    cols = {k: torch.from_numpy(np.ascontiguousarray(a[:, i])).cuda()
            for a, names in ((origins, ("ox", "oy", "oz")), (dirs, ("dx", "dy", "dz"))) for i, k in enumerate(names)}
    out = {k: torch.zeros(n + 64, dtype=getattr(torch, np.dtype(svo.HIT_FIELDS[k]).name), device="cuda") for k in UNCOUNTED}
    for v in out.values():
        v.fill_(0x5A)
    for _ in range(casts):
        p.cast({k: v.data_ptr() for k, v in cols.items()}, {k: v.data_ptr() for k, v in out.items()}, n,
               torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    got = {k: v.cpu().numpy() for k, v in out.items()}
    assert all((v[n:] == 0x5A).all() for v in got.values()), "written past the batch"
    return {k: v[:n] for k, v in got.items()}


@pytest.mark.parametrize("kind,size,dim", [(0, 64, 4), (3, 64, 2), (3, 32, 1), (2, 256, 8), (3, 128, 16)])
def test_mixed_rays_match_the_oracle(oracle_mod, kind, size, dim):
    rng = np.random.default_rng(size + dim)
    o, p = both(oracle_mod, size, dim, svo.gen_scene(kind, size, dim, seed=31, occupancy=0.08, spheres=3, octaves=2,
                                                     base_freq=1.0 / 16, height_lo=2.0, height_hi=size * 0.4))
    origins, dirs = random_rays(rng, size, FLOW + 77)
    at = rng.permutation(len(dirs))[:2500]  # rays for the general forms, and special ones
    dirs[at[:1000]] *= np.float32(1.5)
    dirs[at[1000:1500], 0] = np.nan
    dirs[at[1500:2000]] = np.array([0.0, -0.0, 1.0], np.float32)
    origins[at[2000:]] *= np.float32(1e6)
    ref = o.cast(origins, dirs, threads=16)
    assert_same_hits(device_cast(p, origins, dirs, casts=2), ref, label="mixed %d/%d" % (size, dim))


@pytest.mark.parametrize("n", [1, 31, 33, 4095, 4097, 8192, 65535, GRID - 1, GRID, FLOW - 1, FLOW, FLOW + 1])
def test_sizes_around_the_lines(oracle_mod, n):
    rng = np.random.default_rng(n)
    o, p = both(oracle_mod, 64, 4, svo.gen_scene(0, 64, 4, seed=5, spheres=3, octaves=2, base_freq=1 / 16, height_lo=2.0,
                                                 height_hi=24.0))
    w = 960
    cam = svo.gen_camera_rays([150.0, 90.0, 140.0], [32.0, 16.0, 32.0], 50.0, w, -(-n // w))
    for label, (origins, dirs) in (("random", random_rays(rng, 64, n)), ("camera", (cam[0][:n], cam[1][:n]))):
        ref = o.cast(origins, dirs, threads=16)
        assert_same_hits(device_cast(p, origins, dirs), ref, label="%s %d" % (label, n))


@pytest.mark.parametrize("order", ["random", "camera"])
def test_points_written_over_the_origins(oracle_mod, order):
    """A warp that starts late tells the rays' order from some that are hit points already: each ray is cast once all the same."""
    torch = pytest.importorskip("torch")
    o, p = both(oracle_mod, 64, 4, svo.gen_scene(0, 64, 4, seed=5, spheres=3, octaves=2, base_freq=1 / 16, height_lo=2.0,
                                                 height_hi=24.0))
    n = 3 * FLOW
    if order == "random":
        origins, dirs = random_rays(np.random.default_rng(4), 64, n)
    else:
        origins, dirs = (a[:n] for a in svo.gen_camera_rays([150.0, 90.0, 140.0], [32.0, 16.0, 32.0], 50.0, 1536, 1024))
    ref = o.cast(origins, dirs, threads=16)
    cols = {k: torch.from_numpy(np.ascontiguousarray(a[:, i])).cuda()
            for a, names in ((origins, ("ox", "oy", "oz")), (dirs, ("dx", "dy", "dz"))) for i, k in enumerate(names)}
    status = torch.zeros(n, dtype=torch.uint8, device="cuda")
    p.cast({k: v.data_ptr() for k, v in cols.items()},
           {"status": status.data_ptr(), **{"p" + a: cols["o" + a].data_ptr() for a in "xyz"}}, n,
           torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert np.array_equal(status.cpu().numpy(), ref["status"])
    hit = ref["status"] == 1
    for a in "xyz":
        assert np.array_equal(cols["o" + a].cpu().numpy()[hit].view(np.uint32), ref["p" + a][hit].view(np.uint32)), a


def test_heads_follow_in_place_syncs(oracle_mod):
    rng = np.random.default_rng(9)
    o, p = both(oracle_mod, 64, 4, svo.gen_scene(3, 64, 4, seed=6, occupancy=0.05, spheres=2))
    origins, dirs = random_rays(rng, 64, 20000)
    for k in range(3):
        for pos in rng.integers(0, 64, (200, 3)).tolist():
            for t in (o, p):
                t.clear(pos) if k == 1 else t.insert(pos, 0x11223344 + k, 7)
        p.sync()
        assert_same_hits(p.cast_host(origins, dirs, fields=UNCOUNTED), o.cast(origins, dirs, threads=8), label="sync %d" % k)


@pytest.mark.parametrize("n", [1, 33, 4097, GRID - 1, GRID])
def test_host_buffers_in_place_and_staged(oracle_mod, n):
    rng = np.random.default_rng(n)
    o, p = both(oracle_mod, 64, 4, svo.gen_scene(3, 64, 4, seed=8, occupancy=0.1, spheres=2))
    origins, dirs = random_rays(rng, 64, n)
    ref = o.cast(origins, dirs, threads=16)
    for mode in (0, 1):  # the default, staged copies
        svo.check(svo.lib().svo_set_host_transfer(mode))
        try:
            assert_same_hits(p.cast_host(origins, dirs), ref, counters=True, label="mode %d" % mode)
            assert_same_hits(p.cast_host(origins, dirs, fields=UNCOUNTED), ref, label="uncounted, mode %d" % mode)
        finally:
            svo.check(svo.lib().svo_set_host_transfer(0))
