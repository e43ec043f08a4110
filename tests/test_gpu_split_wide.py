"""Splits of islands around one body with many neighbours: rows on both sides
of what one read holds (8 bodies), bodies met twice in and past the row, and
more waiting bodies than the shared part of the traversal's stack takes
(8160). Every body row (solver set and sleep time among them) and the colours
equal the CPU restatement's, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from forge2d_gb300 import scenes

pytestmark = pytest.mark.gpu


def build(b, count, double, per=100):
    """A floating rack under ``count`` bodies, the first and every
    ``double``-th of them touching it with two shapes; all count as slow from
    the start."""
    slow = dict(type=scenes.DYNAMIC, sleepThreshold=50.0)
    rack = b.create_body(scenes.body_def(**slow))
    half = 0.26 * min(per, count)
    for r in range((count + per - 1) // per):
        b.create_box(rack, scenes.shape_def(density=5.0), half, 0.1, half, 2.0 * r, 1.0, 0.0)
    ids = []
    for k in range(count):
        x, y = 0.26 + 0.52 * (k % per), 2.0 * (k // per) + 0.34
        ids.append(b.create_body(scenes.body_def(positionX=x, positionY=y, **slow)))
        if k % double:
            b.create_circle(ids[-1], scenes.shape_def(), 0.0, 0.0, 0.25)
        else:
            b.create_circle(ids[-1], scenes.shape_def(), -0.12, -0.12, 0.13)
            b.create_circle(ids[-1], scenes.shape_def(), 0.12, -0.12, 0.13)
    return ids


@pytest.mark.parametrize("count,double", [(3, 1), (8, 100), (9, 2), (10, 3), (40, 2), (300, 4), (9100, 50)])
def test_wide_split_equals_port(gpu_lib, count, double):
    from forge2d_gb300.world import GpuWorld
    from oracle.oracle import PortWorld
    wd = scenes.world_def(enableSleep=1, gravityY=0.0)
    g, p = GpuWorld(wd), PortWorld(wd)
    alive = [build(b, count, double) for b in (g, p)]
    slept = False
    for frame in range(40):
        for b, ids in zip((g, p), alive):
            if frame == 4:  # contacts less, so that the island is split once it is slow for long enough
                b.destroy_body(ids[count // 2])
            if frame == 30:
                ball = b.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=0.5, positionY=1.2, linearVelocityY=-10.0))
                b.create_circle(ball, scenes.shape_def(), 0.0, 0.0, 0.2)
            b.step(1.0 / 20.0, 1)
        assert g.sync() == 0
        x, y = g.bodies(), p.bodies()
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), (frame, np.argwhere(x != y)[:4].tolist())
        assert np.array_equal(g.color_counts(), p.color_counts()), frame
        slept = slept or (frame < 30 and g.counters()["awake_bodies"] < count)
    assert slept
    g.close()
    p.close()
