"""The solver's data flow at the sizes where its dealing changes: one part and
several (the limit on bodies with constraints), parts that end inside a
group of 32, bodies shared between parts, overflow constraints and joints
across parts, more substeps than one launch takes. Every body row equals the
CPU restatement's, bit for bit."""
from __future__ import annotations

import os

import numpy as np
import pytest

from forge2d_gb300 import scenes

pytestmark = pytest.mark.gpu

CASES = [
    # (scene, arguments, substeps, frames): pyramids of 378, 406 and 820 bodies lie on both sides of the one-part limit
    ("pyramid", dict(rows=27), 4, 6), ("pyramid", dict(rows=28), 4, 6), ("pyramid", dict(rows=40), 4, 4),
    ("pyramid", dict(rows=2), 1, 8), ("pile", dict(count=33, width=6.0, height=10.0, seed=4), 4, 60),
    ("overflow_heap", dict(platforms=3, per=24, long_count=130, spokes=16), 4, 20),
    ("overflow_heap", dict(platforms=1, per=12, long_count=40, spokes=13), 9, 12),
    ("pyramids_chains", dict(pyramids=3, rows=12, chains=6, links=20), 4, 20),
    ("joint_rigs", dict(copies=9), 17, 6), ("pile", dict(count=700, width=20.0, height=50.0, seed=6), 8, 80),
]


@pytest.mark.parametrize("parts", ["auto", "small"])
@pytest.mark.parametrize("scene,kw,substeps,frames", CASES, ids=["%s-%d-%d" % (c[0], i, c[2]) for i, c in enumerate(CASES)])
def test_parts_equal_port(gpu_lib, scene, kw, substeps, frames, parts):
    from forge2d_gb300.world import GpuWorld
    from oracle.oracle import PortWorld
    wd = scenes.world_def(enableSleep=0)
    if parts == "small":
        os.environ["F2D_NO_CLUSTER_SOLVER"] = "1"
    try:
        g = GpuWorld(wd)
    finally:
        os.environ.pop("F2D_NO_CLUSTER_SOLVER", None)
    p = PortWorld(wd)
    for b in (g, p):
        scenes.build(b, scene, **kw)
    for frame in range(frames):
        g.step(1.0 / 60.0, substeps)
        p.step(1.0 / 60.0, substeps)
        assert g.sync() == 0
        a, b = g.bodies()[:, :9], p.bodies()[:, :9]
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (frame, np.argwhere(a != b)[:4].tolist())
    g.close()
    p.close()
