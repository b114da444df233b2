"""The host-side rules of the casts (shocovox_gb300/csrc/svo_route.h), compiled with the host compiler."""
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
