"""The collide phase at the sizes where its sorts and its colouring change
hands: new pairs of one step on both sides of the block sorts' limits (2048
and 12288 rows), pending colour changes on both sides of what shared memory
holds (3072: two of the three contacts of every triple wait for the first).
Groups of overlapping circles give the counts exactly; contacts, colours and
every body row equal the CPU restatement's, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from forge2d_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sleep", [0, 1])
@pytest.mark.parametrize("members,groups", [(2, 1), (2, 2048), (2, 2049), (2, 12288), (2, 12289), (3, 1536), (3, 1537)])
def test_pair_counts_equal_port(gpu_lib, members, groups, sleep):
    from forge2d_gb300.world import GpuWorld
    from oracle.oracle import PortWorld
    wd = scenes.world_def(enableSleep=sleep)
    g, p = GpuWorld(wd), PortWorld(wd)
    rng = np.random.default_rng(7)
    place = rng.permutation(groups)
    for b in (g, p):
        for k in range(groups):
            x, y = 6.0 * (place[k] % 128), 6.0 * (place[k] // 128)
            for j in range(members):
                body = b.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=x + 0.3 * j, positionY=y + 0.2 * (j & 1)))
                b.create_circle(body, scenes.shape_def(), 0.0, 0.0, 0.5)
    for frame in range(3):
        g.step(1.0 / 60.0, 2)
        p.step(1.0 / 60.0, 2)
        assert g.sync() == 0
        a, b = g.bodies(), p.bodies()
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (frame, np.argwhere(a != b)[:4].tolist())
        assert np.array_equal(g.color_counts(), p.color_counts()), frame
        if frame == 0:
            assert g.counters()["contacts"] == groups * members * (members - 1) // 2
    g.close()
    p.close()
