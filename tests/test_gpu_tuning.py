"""The autotuner compares its candidates, and leaves the world, in the forms of
the step that a long run replays."""
from __future__ import annotations

import pytest

from forge2d_gb300 import scenes

pytestmark = pytest.mark.gpu


def _launches(g, steps):
    out = []
    for _ in range(steps):
        g.step()
        assert g.sync() == 0
        out.append(g.last_step_launches())
    return out


@pytest.mark.parametrize("sleep", [0, 1])
def test_both_forms_are_ready(gpu_lib, sleep):
    from forge2d_gb300.world import GpuWorld
    g = GpuWorld(scenes.world_def(enableSleep=sleep))
    scenes.pyramid(g, rows=10)
    st, chosen, taken = g.autotune(1.0 / 60.0, 4, 1)
    assert st == 0 and taken > 0
    launches = _launches(g, 2 * chosen[1])
    # one step of every period sorts the leaves, the others do not
    assert sorted(set(launches)) == [min(launches), max(launches)] and min(launches) < max(launches)
    assert launches.count(max(launches)) == 2
    g.close()


@pytest.mark.parametrize("rows,stepped,variants", [(10, True, 2), (50, False, 3), (50, True, 3), (60, False, 2), (60, True, 2)])
def test_candidates_differ(gpu_lib, rows, stepped, variants):
    """Up to 400 bodies and above 1600 with constraints, few parts are dealt as
    one per SM: no candidate of their own."""
    from forge2d_gb300.world import GpuWorld
    g = GpuWorld(scenes.world_def(enableSleep=0))
    scenes.pyramid(g, rows=rows)  # 55, 1275 and 1830 boxes
    if stepped:
        for _ in range(3):
            g.step()
    st, chosen, taken = g.autotune(1.0 / 60.0, 4, 1)
    assert st == 0
    assert taken == variants * sum(1 + p for p in (4, 8, 16, 32))
    assert variants == 3 or chosen[0] != 1
    g.close()
