"""Batches without a row layout around the size from which order_kernel tells which of two launches casts them
(kTwoCastsMinRays), against the oracle: both orders, replayed graphs, points over the origins."""
import numpy as np
import pytest

import shocovox_gb300 as svo
from test_gpu_cast import assert_same_hits, both
from test_gpu_flow import device_cast, random_rays

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
TWO = 5 << 19


@pytest.fixture(scope="module")
def scene(oracle_mod):
    return both(oracle_mod, 64, 4, svo.gen_scene(0, 64, 4, seed=5, spheres=3, octaves=2, base_freq=1 / 16, height_lo=2.0,
                                                 height_hi=24.0))


def rays(order, n):
    if order == "random":
        origins, dirs = random_rays(np.random.default_rng(n), 64, n)
        at = np.random.default_rng(1).permutation(n)[:3000]  # a few for the general forms
        dirs[at[:1000]] *= np.float32(1.5)
        dirs[at[1000:2000], 1] = np.nan
        dirs[at[2000:]] = np.array([0.0, -0.0, 1.0], np.float32)
        return origins, dirs
    cam = svo.gen_camera_rays([150.0, 90.0, 140.0], [32.0, 16.0, 32.0], 50.0, 1920, -(-n // 1920))
    return cam[0][:n], cam[1][:n]


@pytest.mark.parametrize("n", [TWO - 1, TWO, TWO + 33])
@pytest.mark.parametrize("order", ["random", "camera"])
def test_both_casts_match_the_oracle(scene, order, n):
    o, p = scene
    origins, dirs = rays(order, n)
    assert_same_hits(device_cast(p, origins, dirs, casts=2), o.cast(origins, dirs, threads=16), label="%s %d" % (order, n))


@pytest.mark.parametrize("order", ["random", "camera"])
def test_points_over_the_origins_and_graphs(scene, order):
    o, p = scene
    n = TWO + 5
    origins, dirs = rays(order, n)
    ref = o.cast(origins, dirs, threads=16)
    host = {k: torch.from_numpy(np.ascontiguousarray(a[:, i])) for a, names in
            ((origins, ("ox", "oy", "oz")), (dirs, ("dx", "dy", "dz"))) for i, k in enumerate(names)}
    cols = {k: v.cuda() for k, v in host.items()}
    status = torch.zeros(n, dtype=torch.uint8, device="cuda")
    hits = {"status": status.data_ptr(), **{"p" + a: cols["o" + a].data_ptr() for a in "xyz"}}
    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        p.cast({k: v.data_ptr() for k, v in cols.items()}, hits, n, stream.cuda_stream)
    hit = ref["status"] == 1
    for k in range(3):
        for name, v in host.items():
            cols[name].copy_(v)
        torch.cuda.synchronize()
        if k == 1:
            p.cast({name: v.data_ptr() for name, v in cols.items()}, hits, n, stream.cuda_stream)
        else:
            graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(status.cpu().numpy(), ref["status"]), k
        for a in "xyz":  # bit for bit, but for a NaN's payload
            got, exp = cols["o" + a].cpu().numpy()[hit], ref["p" + a][hit]
            assert ((got.view(np.uint32) == exp.view(np.uint32)) | (np.isnan(got) & np.isnan(exp))).all(), (k, a)
        status.fill_(9)
