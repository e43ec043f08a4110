"""Island splits on the GPU: the parallel form keeps the reference's order of
bodies, contacts and joints. Scenes whose islands lose contacts and hold
resting bodies, so that splits happen: bodies with more neighbours than one
row holds, joints in the islands, and an island of thousands of bodies. Every
body row (solver set and sleep time among them) equals the CPU restatement's,
bit for bit; a wrong order would show in the sets and colours that follow."""
from __future__ import annotations

import numpy as np
import pytest

from forge2d_gb300 import scenes

pytestmark = pytest.mark.gpu

CASES = [("overflow_heap", dict(platforms=4, per=20, long_count=120, spokes=14), 150, 10),
         ("joint_rigs", dict(copies=4), 200, 20), ("pile", dict(count=60, width=12.0, height=12.0, seed=3), 220, 10),
         ("pile", dict(count=9000, width=300.0, height=40.0, seed=11), 330, 30)]


@pytest.mark.parametrize("scene,kw,frames,every", CASES, ids=["heap", "rigs", "pile60", "pile9000"])
def test_split_equals_port(gpu_lib, scene, kw, frames, every):
    from forge2d_gb300.world import GpuWorld
    from oracle.oracle import PortWorld
    wd = scenes.world_def(enableSleep=1)
    g, p = GpuWorld(wd), PortWorld(wd)
    for b in (g, p):
        scenes.build(b, scene, **kw)
    for frame in range(frames):
        g.step(1.0 / 60.0, 4)
        p.step(1.0 / 60.0, 4)
        if frame % every == every - 1:
            assert g.sync() == 0
            a, b = g.bodies(), p.bodies()
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (frame, np.argwhere(a != b)[:4].tolist())
            assert np.array_equal(g.color_counts(), p.color_counts()), frame
    g.close()
    p.close()
