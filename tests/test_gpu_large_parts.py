"""Sizes past what a block's shared memory holds: a part with more bodies than
row places, and island splits in worlds with more rows than mark bytes.
Equal to the CPU restatement, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from forge2d_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [50, 54])
def test_part_past_its_row_places(gpu_lib, rows):
    """1275 and 1485 boxes in one part, which the tuning's first candidate makes
    of them, on both sides of the 1280 places at 4 substeps."""
    from forge2d_gb300.world import GpuWorld
    from oracle.oracle import PortWorld
    wd = scenes.world_def(enableSleep=0)
    g, p = GpuWorld(wd), PortWorld(wd)
    for b in (g, p):
        scenes.pyramid(b, rows=rows)
    st, _, taken = g.autotune(1.0 / 60.0, 4, 1)
    assert st == 0 and taken == 3 * 64
    for _ in range(taken):
        p.step(1.0 / 60.0, 4)
    x, y = g.bodies()[:, :9], p.bodies()[:, :9]
    assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), np.argwhere(x != y)[:4].tolist()
    g.close()
    p.close()


@pytest.mark.parametrize("singles", [114_000, 115_000])
def test_split_in_a_large_world(gpu_lib, singles):
    """Rows of boxes that split and sleep beside bodies that never sleep, on
    both sides of the 114688 mark bytes."""
    from forge2d_gb300.world import GpuWorld
    from oracle.oracle import PortWorld
    wd = scenes.world_def(enableSleep=1)
    g, p = GpuWorld(wd), PortWorld(wd)
    rows = []
    for b in (g, p):
        ground = b.create_body(scenes.body_def())
        b.create_box(ground, scenes.shape_def(), 100.0, 1.0, 0.0, -1.0, 1.0, 0.0)
        for r in range((singles + 499) // 500):
            b.create_box(ground, scenes.shape_def(), 160.0, 0.1, 400.0, 1.5 * r, 1.0, 0.0)
        for k in range(singles):
            c = b.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=250.0 + 0.6 * (k % 500), positionY=1.5 * (k // 500) + 0.34,
                                              enableSleep=0))
            b.create_circle(c, scenes.shape_def(), 0.0, 0.0, 0.25)
        ids = []
        for k in range(60):
            ids.append(b.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=0.995 * k - 30.0, positionY=0.5, sleepThreshold=50.0)))
            b.create_box(ids[-1], scenes.shape_def(), 0.5, 0.5)
        rows.append(ids)
    for frame in range(30):
        for b, ids in zip((g, p), rows):
            if frame == 4:
                b.destroy_body(ids[20])
            b.step(1.0 / 20.0, 1)
        if frame % 3 == 2:
            assert g.sync() == 0
            x, y = g.bodies(), p.bodies()
            assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), (frame, np.argwhere(x != y)[:4].tolist())
    assert g.counters()["awake_bodies"] == singles  # both halves of the row slept
    g.close()
    p.close()
