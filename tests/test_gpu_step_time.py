"""What a step reports about itself: its launches with those for the proxies
buffered by edits, its device time without the host's captures of the step's
graph."""
from __future__ import annotations

import numpy as np
import pytest

from forge2d_gb300 import scenes

pytestmark = pytest.mark.gpu


def _world():
    from forge2d_gb300.world import GpuWorld
    g = GpuWorld(scenes.world_def(enableSleep=0))
    scenes.pyramid(g, rows=12)
    return g


def test_launches_count_the_buffered_proxies(gpu_lib):
    g = _world()
    g.step()
    counted = {}
    for edits in (0, 1, 0, 32, 0, 33, 0):
        for k in range(edits):
            body = g.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=30.0 + k, positionY=5.0))
            g.create_circle(body, scenes.shape_def(), 0.0, 0.0, 0.3)
        g.step()
        assert g.sync() == 0
        counted.setdefault(edits, g.last_step_launches())
        assert g.last_step_launches() == counted[edits]
    assert counted[1] == counted[32] == counted[0] + 1
    assert counted[33] == counted[0] + 4
    g.close()


def test_step_time_holds_no_capture(gpu_lib):
    """The step is captured at its first step and, without the leaf ordering,
    some twenty steps later; the host needs several steps' time for each."""
    worst = []
    for _ in range(5):
        g = _world()
        ms = []
        for _ in range(40):
            g.step()
            assert g.sync() == 0
            ms.append(g.last_step_ms())
        worst.append(max(ms[4:]) / np.median(ms))
        g.close()
    assert min(worst) < 1.8, worst
