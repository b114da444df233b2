"""The host-side rules of the casts (shocovox_gb300/csrc/svo_route.h, svo_queue.h), compiled with the host compiler."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

import shocovox_gb300 as svo
from shocovox_gb300._lib import Hits, Rays

HERE = os.path.dirname(os.path.abspath(__file__))
RAY = ("ox", "oy", "oz", "dx", "dy", "dz")


@pytest.fixture(scope="module")
def route(tmp_path_factory):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    if shutil.which("g++") is None or not os.path.exists(os.path.join(cuda, "include", "cuda_runtime.h")):
        pytest.skip("needs g++ and the toolkit's headers")
    so = str(tmp_path_factory.mktemp("route") / "route_check.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", os.path.join(cuda, "include"),
                    os.path.join(HERE, "route_check.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


def arrays(rays=0x10000, hits=0x200000, **change):
    """Addresses of six ray arrays and of every hit field, 64 KB apart, but for `change`."""
    at = {k: rays + 0x10000 * i for i, k in enumerate(RAY)}
    at.update({k: hits + 0x10000 * i for i, k in enumerate(svo.HIT_FIELDS)})
    at.update(change)
    return (Rays(*[ctypes.c_void_p(at[k]) for k in RAY]),
            Hits(**{k: ctypes.c_void_p(at[k]) if at[k] else None for k in svo.HIT_FIELDS}))


def test_alignment_of_host_arrays(route):
    def aligned(**change):
        r, h = arrays(**change)
        return route.route_aligned(ctypes.byref(r), ctypes.byref(h)) == 1

    assert aligned()
    assert aligned(**{k: 0 for k in svo.HIT_FIELDS})
    for k in RAY:
        for off in (1, 2, 3):
            assert not aligned(**{k: 0x900000 + off}), (k, off)
    for k, t in svo.HIT_FIELDS.items():
        for off in (1, 2, 3):
            assert aligned(**{k: 0x900000 + off}) == (np.dtype(t).itemsize == 1), (k, off)


def test_overlap_of_host_arrays(route):
    n = 100

    def over(n=n, **change):
        r, h = arrays(**change)
        return route.route_overlap(ctypes.byref(r), ctypes.byref(h), ctypes.c_uint64(n)) == 1

    assert not over() and not over(**{k: 0 for k in svo.HIT_FIELDS})
    at = 0x10000 + 0x10000 * 2  # oz
    for k, t in svo.HIT_FIELDS.items():
        size = np.dtype(t).itemsize
        assert over(**{k: at}) == (size == 1), k  # element for element, or not
        for off in (-size * n + 1, -4, -1, 1, 4, 4 * n - 1):
            assert over(**{k: at + off}) == (-size * n < off), (k, off)
        for off in (-size * n, 4 * n):
            assert not over(**{k: at + off}), (k, off)
        assert not over(0, **{k: at + 4})


CLAIMS = 5


def test_claim_words_of_a_stream_heal(route):
    """A stream's launches one after another each start from a claim word that is 0, whatever an overlap of two of them
    (two streams under one handle) or a replayed graph did before; a captured launch starts from 0 as often as it is replayed."""
    rng = np.random.default_rng(3)

    class Stream:
        def __init__(self):
            self.words, self.turn = [0] * route.route_words(), 0

        def launch(self, captured=False):
            """The steps of a launch's kernel: what it zeroes, and its claims; returns the word it started from."""
            w = route.route_word(self.turn, int(captured))
            self.turn = route.route_launched(self.turn, int(captured))
            return w

        def steps(self, w, start):
            """`start`: gets the value the word had at the first claim."""
            yield self.words.__setitem__(route.route_zeroes(w), 0)
            start.append(self.words[w])
            while True:
                self.words[w] += 1
                if self.words[w] > CLAIMS:
                    break
                yield
            yield

        def run(self, captured=False):
            w, start = self.launch(captured), []
            if captured:
                self.words[w] = 0  # the graph's memset node
            for _ in self.steps(w, start):
                pass
            return start[0]

    for _ in range(300):
        s = Stream()
        for _ in range(rng.integers(0, 4)):
            assert s.run() == 0
        # two launches overlap, their steps in any order
        both = [s.steps(s.launch(), []) for _ in range(2)]
        while both:
            k = int(rng.integers(len(both)))
            if next(both[k], StopIteration) is StopIteration:
                both.pop(k)
        s.run()  # the one after them may find a word that one of them was still counting in
        for _ in range(4):
            if rng.integers(2):
                assert s.run(captured=True) == 0
            assert s.run() == 0


@pytest.mark.parametrize("gap", [1, 2, 7, 65536])
def test_spans_of_changed_nodes(route, gap):
    """All runs and nothing else but what lies between runs fewer than `gap` apart."""
    rng = np.random.default_rng(gap)
    for case in range(200):
        ends = np.sort(rng.choice(400, 2 * int(rng.integers(0, 30)), replace=False)).astype(np.uint64)
        runs = np.ascontiguousarray(ends.reshape(-1, 2))
        out = np.zeros((len(runs) + 1, 2), np.uint64)
        k = route.route_spans(runs.ctypes.data_as(ctypes.c_void_p), ctypes.c_uint64(len(runs)), ctypes.c_uint64(gap),
                              out.ctypes.data_as(ctypes.c_void_p))
        covered = np.zeros(400, bool)
        for a, b in runs.tolist():
            covered[a:b] = True
        at = np.nonzero(covered)[0].tolist()
        expected = []
        for i in at:
            if expected and i - expected[-1][1] < gap:
                expected[-1][1] = i + 1
            else:
                expected.append([i, i + 1])
        assert out[:k].tolist() == expected, case
