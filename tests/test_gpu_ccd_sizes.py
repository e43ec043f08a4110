"""Continuous collision at the static counts where its search changes: a
thread's scan (up to 64 static shapes), a warp's scan (up to 1024), the pair
tree's walk. Fast bodies of one and two shapes pass rows of boxes; every
body row equals the CPU restatement's, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from forge2d_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("statics", [1, 64, 65, 128, 129, 1024, 1025])
def test_fast_bodies_equal_port(gpu_lib, statics):
    from forge2d_gb300.world import GpuWorld
    from oracle.oracle import PortWorld
    wd = scenes.world_def(enableSleep=0)
    g, p = GpuWorld(wd), PortWorld(wd)
    for b in (g, p):
        rng = np.random.default_rng(5)
        ground = b.create_body(scenes.body_def(type=scenes.STATIC))
        for k in range(statics):
            x, y = 0.8 * (k % 96) - 38.0, -1.5 * (k // 96)
            b.create_box(ground, scenes.shape_def(), 0.3 + 0.1 * (k % 2), 0.05, x, y, 1.0, 0.0, 0.0)
        for k in range(70):
            body = b.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=float(rng.uniform(-38.0, 38.0)), positionY=float(rng.uniform(2.0, 6.0)),
                                                 linearVelocityX=float(rng.uniform(-90.0, 90.0)), linearVelocityY=float(rng.uniform(-300.0, -60.0)),
                                                 angularVelocity=float(rng.uniform(-9.0, 9.0)), isBullet=k % 3 == 0))
            if k % 2:
                b.create_circle(body, scenes.shape_def(), 0.0, 0.0, 0.15)
            else:
                b.create_box(body, scenes.shape_def(), 0.15, 0.25)
            if k % 5 == 0:
                b.create_circle(body, scenes.shape_def(), 0.2, 0.1, 0.1)
    for frame in range(6):
        g.step(1.0 / 60.0, 4)
        p.step(1.0 / 60.0, 4)
        assert g.sync() == 0
        x, y = g.bodies()[:, :9], p.bodies()[:, :9]
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), (frame, np.argwhere(x != y)[:4].tolist())
    g.close()
    p.close()
