"""Bodies created, edited and destroyed between steps at the counts where
their rows change from one launch to several and to whole-array copies (8
and 32 rows, 32 buffered moves), and box and ray queries on both sides of the
list that reaches the host directly (2048 shapes). Everything equals the CPU
restatement's, body rows bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from forge2d_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sleep", [0, 1])
@pytest.mark.parametrize("count", [1, 8, 9, 32, 33])
def test_edited_rows_equal_port(gpu_lib, count, sleep):
    from forge2d_gb300.world import GpuWorld
    from oracle.oracle import PortWorld
    wd = scenes.world_def(enableSleep=sleep)
    g, p = GpuWorld(wd), PortWorld(wd)
    alive = [list(scenes.pile(b, count=120, width=16.0, height=24.0, seed=9)) for b in (g, p)]
    for frame in range(12):
        for b, ids in zip((g, p), alive):
            if frame % 3 == 1:
                for k in range(count):
                    b.destroy_body(ids.pop(0))
                    body = b.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=-7.0 + 0.4 * k, positionY=25.0 + frame))
                    b.create_circle(body, scenes.shape_def(), 0.0, 0.0, 0.3)
                    b.create_box(body, scenes.shape_def(), 0.2, 0.4)
                    ids.append(body)
            b.step(1.0 / 60.0, 4)
        assert g.sync() == 0
        x, y = g.bodies()[:, :9], p.bodies()[:, :9]
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), (frame, np.argwhere(x != y)[:4].tolist())
    g.close()
    p.close()


@pytest.mark.parametrize("count", [1, 2048, 2049])
def test_queries_equal_port(gpu_lib, count):
    from forge2d_gb300.world import GpuWorld
    from oracle.oracle import PortWorld
    wd = scenes.world_def(enableSleep=0)
    g, p = GpuWorld(wd), PortWorld(wd)
    place = np.random.default_rng(count).permutation(count)
    for b in (g, p):
        for k in range(count):
            body = b.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=3.0 * (place[k] % 64), positionY=3.0 * (place[k] // 64)))
            b.create_circle(body, scenes.shape_def(), 0.0, 0.0, 0.5)
    for box in [(-10.0, -10.0, 400.0, 400.0), (500.0, 500.0, 501.0, 501.0), (-1.0, -1.0, 4.0, 4.0)] * 2:
        a, b = g.overlap_aabb(*box), p.overlap_aabb(*box)
        assert sorted(np.asarray(a).ravel().tolist()) == sorted(np.asarray(b).ravel().tolist()), box
    for ray in [(-5.0, 0.0, 500.0, 0.0), (-5.0, -2.0, 500.0, 0.0), (-5.0, 0.3, 300.0, 90.0)] * 2:
        a, b = g.cast_ray_closest(*ray), p.cast_ray_closest(*ray)
        assert str(a) == str(b), ray
    g.close()
    p.close()


@pytest.mark.parametrize("edit", [14, 15, 16, 17, 24])
def test_replayed_forms_equal_port(gpu_lib, edit):
    """The step is replayed in two forms, with and without the leaf ordering,
    the second from the 16th unchanged step that sorts nothing: an edit around
    there, and a change of the substeps after it."""
    from forge2d_gb300.world import GpuWorld
    from oracle.oracle import PortWorld
    wd = scenes.world_def(enableSleep=0)
    g, p = GpuWorld(wd), PortWorld(wd)
    for b in (g, p):
        scenes.build(b, "pile", count=60, width=12.0, height=12.0, seed=3)
    for frame in range(60):
        for b in (g, p):
            if frame == edit:
                body = b.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=0.5, positionY=14.0))
                b.create_circle(body, scenes.shape_def(), 0.0, 0.0, 0.3)
            b.step(1.0 / 60.0, 4 if frame < edit + 25 else 3)
        assert g.sync() == 0
        x, y = g.bodies()[:, :9], p.bodies()[:, :9]
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), (frame, np.argwhere(x != y)[:4].tolist())
    g.close()
    p.close()
