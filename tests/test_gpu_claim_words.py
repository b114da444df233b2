"""Claim words of the queued casts across launches: graphs replayed beside casts on the stream they were captured on, and
casts after an overlap that include/svo.h rules out (two graphs of one stream at once), which may spoil those two only."""
import ctypes

import numpy as np
import pytest

import shocovox_gb300 as svo
from test_gpu_cast import assert_same_hits, both
from test_gpu_flow import FLOW, UNCOUNTED, random_rays

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def scene(oracle_mod):
    return both(oracle_mod, 64, 4, svo.gen_scene(0, 64, 4, seed=5, spheres=3, octaves=2, base_freq=1 / 16, height_lo=2.0,
                                                 height_hi=24.0))


class Call:
    """One cast on device buffers: through svo_cast (`row`), or the batched cast's unordered items."""

    def __init__(self, scene, kind, seed):
        o, self.p = scene
        if kind == "rows":
            origins, dirs = svo.gen_camera_rays([150.0, 90.0, 140.0 + seed], [32.0, 16.0, 32.0], 50.0, 431, 331)
        else:
            origins, dirs = random_rays(np.random.default_rng(seed), 64, FLOW + 5 if kind == "plain" else 30011)
        self.n, self.row = len(origins), 431 if kind == "rows" else 0
        self.ref = o.cast(origins, dirs, threads=16)
        self.rays = {k: torch.from_numpy(np.ascontiguousarray(a[:, i])).cuda()
                     for a, names in ((origins, ("ox", "oy", "oz")), (dirs, ("dx", "dy", "dz"))) for i, k in enumerate(names)}
        self.out = {k: torch.zeros(self.n, dtype=getattr(torch, np.dtype(svo.HIT_FIELDS[k]).name), device="cuda")
                    for k in UNCOUNTED}
        self.ws = svo.BatchWorkspace() if kind.startswith("items") else None
        self.cfg = svo.LaunchConfig(0, 0, 0, 0, 1, 0, 0)
        self.parts = int(kind[5:]) if self.ws else 0

    def run(self, stream):
        r, h = ({k: v.data_ptr() for k, v in d.items()} for d in (self.rays, self.out))
        if not self.ws:
            return self.p.cast(r, h, self.n, stream.cuda_stream, self.row)
        ends = [self.n * k // self.parts for k in range(self.parts + 1)]
        at = lambda d, a: {k: v.data_ptr() + a * v.element_size() for k, v in d.items()}  # noqa: E731
        self.ws.cast([(self.p, at(self.rays, a), b - a, at(self.out, a)) for a, b in zip(ends, ends[1:])], self.cfg,
                     stream.cuda_stream)

    def clear(self):
        for v in self.out.values():
            v.fill_(0x5A)
        torch.cuda.synchronize()

    def check(self, label):
        torch.cuda.synchronize()
        assert_same_hits({k: v.cpu().numpy() for k, v in self.out.items()}, self.ref, label=label)
        self.clear()


def captured(call, stream):
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        call.run(stream)
    return g


@pytest.mark.parametrize("kind", ["rows", "plain", "items1", "items3"])
def test_graphs_beside_casts_on_their_stream(scene, kind):
    s, other = torch.cuda.Stream(), torch.cuda.Stream()
    graphed, direct = Call(scene, kind, 1), Call(scene, kind, 2)
    graphed.run(s)  # sizes the workspace
    torch.cuda.synchronize()
    g = captured(graphed, s)
    for c in (graphed, direct):
        c.clear()
    for k in range(5):
        with torch.cuda.stream(other):
            g.replay()
        direct.run(s)
        if k % 2:
            direct.run(s)
        graphed.check("replay %d" % k)
        direct.check("direct %d" % k)


def test_casts_after_two_graphs_of_a_stream_overlapped(scene):
    s, streams = torch.cuda.Stream(), (torch.cuda.Stream(), torch.cuda.Stream())
    calls = [Call(scene, "rows", 1), Call(scene, "plain", 2)]
    graphs = [captured(c, s) for c in calls]
    direct = Call(scene, "plain", 3)
    for _ in range(10):
        for g, st in zip(graphs, streams):
            with torch.cuda.stream(st):
                g.replay()
    torch.cuda.synchronize()
    direct.clear()
    for c in calls:
        c.clear()
    for k in range(3):
        direct.run(s)
        direct.check("direct %d" % k)
        for c, g in zip(calls, graphs):
            with torch.cuda.stream(s):
                g.replay()
            c.check("replay %d" % k)


def test_workspace_creation_leaves_the_default_stream_alone():
    """It neither waits for work that the default stream has queued nor ends a capture that the stream must not touch."""
    svo.BatchWorkspace()
    torch.cuda.synchronize()
    busy = torch.cuda.Event()
    torch.cuda._sleep(400_000_000)  # about 0.2 s
    busy.record()
    ws = svo.BatchWorkspace()
    assert not busy.query()
    busy.synchronize()
    rt = ctypes.CDLL("libcudart.so.13")
    st, graph = ctypes.c_void_p(), ctypes.c_void_p()
    assert rt.cudaStreamCreate(ctypes.byref(st)) == 0  # one that the default stream waits for
    assert rt.cudaStreamBeginCapture(st, 2) == 0  # relaxed: allocations are allowed meanwhile
    try:
        other = svo.BatchWorkspace()
    finally:
        rc = rt.cudaStreamEndCapture(st, ctypes.byref(graph))
    assert rc == 0
    assert rt.cudaGraphDestroy(graph) == 0 and rt.cudaStreamDestroy(st) == 0
    del ws, other
