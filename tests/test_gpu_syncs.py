"""In-place syncs of a scene of many nodes: the heads that casts read follow edits far apart and close together, and a
fresh upload of the edited scene is cast the same."""
import numpy as np
import pytest

import shocovox_gb300 as svo
from helpers import COMPLEX, INSERT, ops_from
from test_gpu_cast import assert_same_hits, both
from test_gpu_flow import UNCOUNTED, random_rays

pytestmark = pytest.mark.gpu


def test_heads_of_changed_nodes_only(oracle_mod):
    rng = np.random.default_rng(12)
    S = 2048
    pts = rng.integers(0, S, (40_000, 3))
    o, p = both(oracle_mod, S, 2, ops_from([(INSERT, int(x), int(y), int(z), COMPLEX, 0x11223300 + i % 200, i + 1)
                                            for i, (x, y, z) in enumerate(pts)]))
    assert p.stats()["nodes"] > 2 << 16  # changed nodes can lie more than a launch's gap apart
    origins, dirs = random_rays(rng, S, 60_000)
    aimed = pts[rng.integers(0, len(pts), 40_000)] + np.float32(0.5) - origins[:40_000]
    dirs[:40_000] = (aimed / np.sqrt((aimed * aimed).sum(1, keepdims=True))).astype(np.float32)
    for step, edits in enumerate((pts[:1], pts[[0, 1, 20_000, 39_999]], pts[100:400], rng.integers(0, S, (300, 3)))):
        for pos in edits.tolist():
            for t in (o, p):
                t.clear(pos) if step < 3 else t.insert(pos, 0x55667788, 3)
        p.sync()
        ref = o.cast(origins, dirs, threads=16)
        assert_same_hits(p.cast_host(origins, dirs, fields=UNCOUNTED), ref, label="sync %d" % step)
    p.upload()
    assert_same_hits(p.cast_host(origins, dirs, fields=UNCOUNTED), ref, label="upload")
