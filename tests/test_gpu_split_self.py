"""A split of an island whose bodies have joints to themselves: the joints
stay with their bodies' islands, go to sleep and wake with them. Body rows
(solver set and sleep time among them), colours and joint reactions equal the
CPU restatement's, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from forge2d_gb300 import scenes

pytestmark = pytest.mark.gpu


def _build(b, boxes):
    """Boxes side by side on the ground, slow enough for sleep at once; every
    second one has a joint to itself, two of them a joint to each other."""
    ground = b.create_body(scenes.body_def(positionY=-1.0))
    b.create_box(ground, scenes.shape_def(), 100.0, 1.0)
    ids, joints = [], []
    for k in range(boxes):
        ids.append(b.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=0.995 * k, positionY=0.5, sleepThreshold=50.0)))
        b.create_box(ids[-1], scenes.shape_def(), 0.5, 0.5)
    for k in range(0, boxes, 2):
        for _ in range(1 + k % 3):
            joints.append((k, b.create_joint(scenes.joint_def(type=scenes.JOINT_MOUSE, bodyA=ids[k], bodyB=ids[k], hertz=2.0, dampingRatio=0.7,
                                                          maxForce=2.0, targetX=0.995 * k, targetY=0.6))))
    b.create_revolute(scenes.revolute_def(bodyA=ids[0], bodyB=ids[1], localAnchorAX=0.5, localAnchorBX=-0.495))
    return ids, joints


@pytest.mark.parametrize("boxes", [3, 12, 40])
def test_split_keeps_self_joints(gpu_lib, boxes):
    from forge2d_gb300.world import GpuWorld
    from oracle.oracle import PortWorld
    wd = scenes.world_def(enableSleep=1)
    g, p = GpuWorld(wd), PortWorld(wd)
    built = [_build(b, boxes) for b in (g, p)]
    asleep = 0
    for frame in range(120):
        for b, (ids, joints) in zip((g, p), built):
            if frame == 10:  # a contact less, so that the island is split when it is slow for long enough
                b.destroy_body(ids[boxes // 2])
            if frame == 80:  # wakes the first half
                ball = b.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=0.2, positionY=3.0, linearVelocityY=-20.0))
                b.create_circle(ball, scenes.shape_def(), 0.0, 0.0, 0.3)
            b.step(1.0 / 60.0, 4)
        assert g.sync() == 0
        x, y = g.bodies(), p.bodies()
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), (frame, np.argwhere(x != y)[:4].tolist())
        assert np.array_equal(g.color_counts(), p.color_counts()), frame
        for (owner, a), (_, b) in zip(built[0][1], built[1][1]):
            if frame < 10 or owner != boxes // 2:
                assert np.array_equal(np.asarray(g.joint_constraint(a)), np.asarray(p.joint_constraint(b))), frame
        asleep = max(asleep, boxes - 1 - g.counters()["awake_bodies"])
    assert asleep > 0  # the halves slept
    g.close()
    p.close()
