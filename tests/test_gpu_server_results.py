"""Where a server's results go: pageable arrays at any address (the copy kernel's 16-, 4- and 1-byte paths), page-locked ones
(copy engines), both in one batch, and batches of more cameras and more pieces than one launch takes."""
import numpy as np
import pytest

import shocovox_gb300 as svo
from test_gpu_host_arrays import shifted
from test_gpu_server import FIELDS, expected, out_arrays, same, scenes

pytestmark = pytest.mark.gpu
SIZES = [(160, 120), (1, 1), (7, 5), (64, 48), (33, 1), (1283, 3)]  # bytes of a field from 1 up, odd ones among them


def requests(sc, n):
    rng = np.random.default_rng(n)
    reqs = []
    for i in range(n):
        j = i % len(sc)
        S, a = float(sc[j].size), rng.uniform(0, 2 * np.pi)
        reqs.append((j, [S / 2 + 1.5 * S * np.cos(a), 1.1 * S, S / 2 + 1.5 * S * np.sin(a)], [S / 2, S / 3, S / 2], 60.0) +
                    SIZES[i % len(SIZES)])
    return reqs


def serve(sc, reqs, outs, **config):
    """All requests behind a large one, so that the server finds them waiting together; returns the largest batch."""
    srv = svo.Server(max_inflight=1, max_batch_requests=128, **config)
    try:
        for t in sc:
            srv.add_scene(t)
        first = srv.submit(0, [100.0, 90.0, 100.0], [32.0, 20.0, 32.0], 60.0, 8192, 4096,
                           out={"status": np.zeros(8192 * 4096, np.uint8)})
        ids = [srv.submit(*r, out=o) for r, o in zip(reqs, outs)]
        srv.wait(first)
        return max(srv.wait(i)["batch_requests"] for i in ids)
    finally:
        srv.close()


@pytest.mark.parametrize("offset", [0, 1, 2, 3, 4, 8, 12, 15])
def test_results_at_any_address(offset):
    sc = scenes()
    reqs = requests(sc, 12)
    refs = [expected(sc, r) for r in reqs]
    outs = [{k: shifted(v, offset) for k, v in out_arrays(r[4], r[5]).items()} for r in reqs]
    serve(sc, reqs, outs)
    for got, ref in zip(outs, refs):
        same(got, ref)


def test_more_cameras_and_pieces_than_one_launch_takes():
    sc = scenes()
    reqs = requests(sc, 120)  # 120 cameras (32 a launch), 1,440 pieces (128 a launch)
    refs = [expected(sc, r) for r in reqs]
    outs = [out_arrays(r[4], r[5]) for r in reqs]
    assert serve(sc, reqs, outs) > 33
    for got, ref in zip(outs, refs):
        same(got, ref)


def test_page_locked_and_pageable_results_in_one_batch():
    torch = pytest.importorskip("torch")
    sc = scenes()
    reqs = requests(sc, 36)
    refs = [expected(sc, r) for r in reqs]
    outs, keep = [], []
    for i, r in enumerate(reqs):
        out = out_arrays(r[4], r[5])
        for k in FIELDS[i % 3::3]:  # a third of the fields of each request
            t = torch.zeros(out[k].nbytes, dtype=torch.uint8).pin_memory()
            keep.append(t)
            out[k] = t.numpy().view(out[k].dtype)
        outs.append(out)
    serve(sc, reqs, outs)
    for got, ref in zip(outs, refs):
        same(got, ref)
