"""Moving, turning bodies of several shapes disabled and enabled again: their
rows, the centre of mass among them, equal the CPU restatement's, bit for
bit."""
from __future__ import annotations

import numpy as np
import pytest

from forge2d_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sleep", [0, 1])
def test_disabled_bodies_keep_their_centre(gpu_lib, sleep):
    from forge2d_gb300.world import GpuWorld
    from oracle.oracle import PortWorld
    wd = scenes.world_def(enableSleep=sleep)
    g, p = GpuWorld(wd), PortWorld(wd)
    made = []
    for b in (g, p):
        rng = np.random.default_rng(6)
        ids = []
        for k in range(40):
            ids.append(b.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=2.0 * k, positionY=float(rng.uniform(1.0, 9.0)),
                                                     linearVelocityX=float(rng.normal()), angularVelocity=float(rng.normal(0.0, 4.0)))))
            b.create_box(ids[-1], scenes.shape_def(), 0.3, 0.2, 0.1 + 0.01 * k, -0.05, 1.0, 0.0)
            b.create_circle(ids[-1], scenes.shape_def(density=3.0), -0.2, 0.15, 0.2)
        made.append(ids)
    for frame in range(24):
        for b, ids in zip((g, p), made):
            for k in range(40):
                if frame == 2 + k % 7:
                    b.body_disable(ids[k])
                elif frame == 10 + k % 5:
                    b.body_enable(ids[k])
            b.step(1.0 / 60.0, 4)
        assert g.sync() == 0
        x, y = g.bodies()[:, :9], p.bodies()[:, :9]
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), (frame, np.argwhere(x != y)[:4].tolist())
    g.close()
    p.close()
