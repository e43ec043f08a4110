"""Joints whose two ends are the same body, in a graph colour and in the
overflow array, alone on a body and among its other constraints. Every body
row and joint reaction equals the CPU restatement's, bit for bit."""
from __future__ import annotations

import math

import numpy as np
import pytest

from forge2d_gb300 import scenes

pytestmark = pytest.mark.gpu

TYPES = {"revolute": None, "weld": 2, "distance": 3, "prismatic": 4, "wheel": 5, "motor": 6, "mouse": 7, "filter": 8}


def _self_joint(b, kind, body, x, y):
    if kind == "revolute":
        return b.create_revolute(scenes.revolute_def(bodyA=body, bodyB=body, localAnchorAX=0.2, localAnchorBX=-0.1, enableSpring=1,
                                                     hertz=2.0, dampingRatio=0.5, enableMotor=1, motorSpeed=1.0, maxMotorTorque=3.0))
    return b.create_joint(scenes.joint_def(type=TYPES[kind], bodyA=body, bodyB=body, localAnchorAX=0.2, localAnchorBX=-0.1,
                                           localAnchorBY=0.15, linearHertz=3.0, angularHertz=2.0, linearDampingRatio=0.7,
                                           length=0.3, enableSpring=1, hertz=4.0, dampingRatio=0.6, maxForce=400.0,
                                           maxTorque=10.0, targetX=x + 2.0, targetY=y + 1.5))


def _build(b, kind, spokes):
    """A free body, a box in a stack and a hub of revolute spokes, each with
    two joints to itself; with 13 spokes the hub's lie past the colours."""
    ground = b.create_body(scenes.body_def(positionY=-1.0))
    b.create_box(ground, scenes.shape_def(), 40.0, 1.0)
    joints = []
    free = b.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=-12.0, positionY=6.0, angularVelocity=1.0))
    b.create_box(free, scenes.shape_def(), 0.4, 0.3)
    stack = []
    for k in range(6):
        stack.append(b.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=-5.0 + 0.05 * k, positionY=0.5 + k)))
        b.create_box(stack[-1], scenes.shape_def(restitution=0.2), 0.5, 0.5)
    hub = b.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=4.0, positionY=4.0))
    b.create_circle(hub, scenes.shape_def(), 0.0, 0.0, 0.5)
    for k in range(spokes):
        a = 2.0 * math.pi * k / spokes
        s = b.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=4.0 + 1.5 * math.cos(a), positionY=4.0 + 1.5 * math.sin(a),
                                          rotationCos=math.cos(a), rotationSin=math.sin(a)))
        b.create_box(s, scenes.shape_def(), 0.3, 0.15)
        b.create_revolute(scenes.revolute_def(bodyA=hub, bodyB=s, localAnchorBX=-1.5, enableSpring=1, hertz=4.0, dampingRatio=0.5))
    for body, x, y in ((free, -12.0, 6.0), (stack[2], -5.0, 2.5), (hub, 4.0, 4.0)):
        for k in range(2):
            joints.append(_self_joint(b, kind, body, x + k, y))
    return joints


@pytest.mark.parametrize("sleep", [0, 1])
@pytest.mark.parametrize("spokes", [3, 13])
@pytest.mark.parametrize("kind", sorted(TYPES))
def test_self_joints_equal_port(gpu_lib, kind, spokes, sleep):
    from forge2d_gb300.world import GpuWorld
    from oracle.oracle import PortWorld
    wd = scenes.world_def(enableSleep=sleep)
    g, p = GpuWorld(wd), PortWorld(wd)
    jg, jp = (_build(b, kind, spokes) for b in (g, p))
    for frame in range(24):
        g.step(1.0 / 60.0, 4)
        p.step(1.0 / 60.0, 4)
        assert g.sync() == 0
        a, b = g.bodies()[:, :9], p.bodies()[:, :9]
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (frame, np.argwhere(a != b)[:4].tolist())
    assert np.isfinite(a).all()
    for x, y in zip(jg, jp):
        f, h = np.asarray(g.joint_constraint(x), np.float32), np.asarray(p.joint_constraint(y), np.float32)
        assert np.array_equal(f, h), (kind, f, h)
    g.close()
    p.close()


@pytest.mark.parametrize("sleep", [0, 1])
def test_destroyed_body_frees_its_self_joint_once(gpu_lib, sleep):
    """Two joints made after it have different ids, and the world goes on as
    one in which the joint was destroyed first."""
    from forge2d_gb300.world import GpuWorld
    worlds = []
    for first in (True, False):
        g = GpuWorld(scenes.world_def(enableSleep=sleep))
        ground = g.create_body(scenes.body_def(positionY=-1.0))
        g.create_box(ground, scenes.shape_def(), 20.0, 1.0)
        ids = []
        for k in range(6):
            ids.append(g.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=1.1 * k, positionY=2.0)))
            g.create_box(ids[-1], scenes.shape_def(), 0.5, 0.5)
        joint = _self_joint(g, "mouse", ids[2], 2.2, 2.0)
        for _ in range(5):
            g.step()
        if first:
            g.destroy_joint(joint)
        g.destroy_body(ids[2])
        a = g.create_revolute(scenes.revolute_def(bodyA=ids[0], bodyB=ids[1], localAnchorAX=0.55, localAnchorBX=-0.55))
        b = g.create_revolute(scenes.revolute_def(bodyA=ids[3], bodyB=ids[4], localAnchorAX=0.55, localAnchorBX=-0.55))
        assert a[0] != b[0]
        for _ in range(30):
            g.step()
        assert g.sync() == 0 and g.counters()["joints"] == 2
        worlds.append(g)
    x, y = (g.bodies()[:, :9] for g in worlds)
    assert np.array_equal(x.view(np.uint32), y.view(np.uint32))
    for g in worlds:
        g.close()
