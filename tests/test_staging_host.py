"""The batched cast's share-out of staged records (assign_staging, shocovox_gb300/csrc/svo_batch.cu), on the host."""
import ctypes
import glob
import os
import shutil
import subprocess

import numpy as np
import pytest

import shocovox_gb300 as svo  # noqa: F401  (builds the objects)

HERE = os.path.dirname(os.path.abspath(__file__))
LIB = os.path.join(os.path.dirname(HERE), "shocovox_gb300", "_lib")
RECORDS = 768  # a block's


@pytest.fixture(scope="module")
def stage(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("needs nvcc")
    so = str(tmp_path_factory.mktemp("stage") / "stage_check.so")
    objects = [o for o in glob.glob(os.path.join(LIB, "*.o")) if not o.endswith("svo_batch.o")]
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O1", "-std=c++17", "-fmad=false", "-Xcompiler",
                    "-fPIC,-O1", "-shared", os.path.join(HERE, "stage_check.cu")] + objects +
                   ["-o", so, "-lpthread", "-ldl"], check=True, capture_output=True)
    lib = ctypes.CDLL(so)

    def run(scene, n, records):
        scene, n, records = np.array(scene, np.uint32), np.array(n, np.uint64), np.array(records, np.uint32)
        out = np.zeros((len(scene), 3), np.uint32)
        vp = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
        total = lib.stage_check(ctypes.c_uint32(len(scene)), vp(scene), vp(n), ctypes.c_uint32(len(records)), vp(records), vp(out))
        return total, out.tolist()

    return run


def test_scenes_in_claim_order_share_the_records(stage):
    total, got = stage([0, 1, 0, 2], [5, 5, 5, 5], [100, 200, 300])
    assert total == 600 and got == [[0, 100, 1], [100, 200, 1], [0, 100, 0], [300, 300, 1]]
    total, got = stage([0, 1, 2], [5, 5, 5], [500, 300, 200])  # the second does not fit, the third does
    assert total == 700 and got == [[0, 500, 1], [0, 0, 0], [500, 200, 1]]


def test_items_cast_apart_take_no_records(stage):
    """Items without rays in claim order (unordered or empty ones) neither stage their scene nor take others' share."""
    total, got = stage([0, 1], [0, 5], [RECORDS, 300])
    assert total == 300 and got == [[0, 0, 0], [0, 300, 1]]
    total, got = stage([0, 1, 0, 1], [0, 0, 5, 5], [200, 300])  # staged for the first item that has such rays
    assert total == 500 and got == [[0, 0, 0], [0, 0, 0], [0, 200, 1], [200, 300, 1]]
    assert stage([0, 1], [0, 0], [200, 300]) == (0, [[0, 0, 0], [0, 0, 0]])
