"""Sleeping bodies that gain or lose a shape and are then woken by a touch
inside a step: their old contacts are solved with the new masses. Body rows
equal the CPU restatement's, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from forge2d_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edit", ["gain", "lose"])
def test_woken_contacts_have_the_present_mass(gpu_lib, edit):
    from forge2d_gb300.world import GpuWorld
    from oracle.oracle import PortWorld
    wd = scenes.world_def(enableSleep=1)
    g, p = GpuWorld(wd), PortWorld(wd)
    made = []
    for b in (g, p):
        ground = b.create_body(scenes.body_def(positionY=-1.0))
        b.create_box(ground, scenes.shape_def(), 60.0, 1.0)
        rows = []
        for k in range(12):
            body = b.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=4.0 * k, positionY=0.5, sleepThreshold=5.0))
            b.create_box(body, scenes.shape_def(), 0.5, 0.5)
            rows.append((body, b.create_circle(body, scenes.shape_def(density=4.0), 0.2, 0.3, 0.3)))
        made.append(rows)
    asleep = 0
    for frame in range(90):
        for b, rows in zip((g, p), made):
            for k, (body, extra) in enumerate(rows):
                if frame == 45 and edit == "gain":
                    b.create_circle(body, scenes.shape_def(density=6.0), -0.3, 0.4, 0.25 + 0.01 * k)
                elif frame == 45:
                    b.destroy_shape(extra)
                if frame == 46:
                    ball = b.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=4.0 * k + 0.05 * k, positionY=4.0,
                                                         linearVelocityY=-14.0))
                    b.create_circle(ball, scenes.shape_def(density=2.0), 0.0, 0.0, 0.3)
            b.step(1.0 / 60.0, 4)
        assert g.sync() == 0
        x, y = g.bodies(), p.bodies()
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), (frame, np.argwhere(x != y)[:4].tolist())
        asleep = max(asleep, 12 - g.counters()["awake_bodies"]) if frame < 46 else asleep
    assert asleep == 12
    g.close()
    p.close()
