"""One body under many others: its overflow constraints at the counts where
the set-up of their ranks and their order changes hands (256 of a body, 1024
of a part), from contacts and from joints. Every body row equals the CPU
restatement's, bit for bit."""
from __future__ import annotations

import math
import os

import numpy as np
import pytest

from forge2d_gb300 import scenes

pytestmark = pytest.mark.gpu


def shelves(b, count, body_type=scenes.DYNAMIC, head="corner", per=100, restitution=True):
    """``count`` circles on one body that is a rack of shelves, a third of them
    with restitution. ``head`` is where the rack's place in the spatial order
    lies: in the corner (its constraints then make one part) or in the middle."""
    rack = b.create_body(scenes.body_def(type=body_type, linearVelocityY=0.5))
    rows = (count + per - 1) // per
    half = 0.26 * min(per, count)
    order = list(range(rows))
    order.append(order.pop(0 if head == "corner" else rows // 2))  # the last shape made leads the body's list
    for r in order:
        b.create_box(rack, scenes.shape_def(), half if r or head != "corner" else half + 2.0, 0.1,
                     half if r or head != "corner" else half - 2.0, 2.0 * r, 1.0, 0.0)
    for k in range(count):
        c = b.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=0.26 + 0.52 * (k % per), positionY=2.0 * (k // per) + 0.34))
        b.create_circle(c, scenes.shape_def(restitution=0.3 if restitution and k % 3 == 0 else 0.0), 0.0, 0.0, 0.25)


def spokes(b, count):
    hub = b.create_body(scenes.body_def(type=scenes.DYNAMIC))
    b.create_circle(hub, scenes.shape_def(density=20.0), 0.0, 0.0, 0.5)
    for k in range(count):
        a = 2.0 * math.pi * k / count
        r = 0.12 * count
        s = b.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=r * math.cos(a), positionY=r * math.sin(a),
                                          rotationCos=math.cos(a), rotationSin=math.sin(a)))
        b.create_box(s, scenes.shape_def(), 0.3, 0.15)
        b.create_revolute(scenes.revolute_def(bodyA=hub, bodyB=s, localAnchorBX=-r, enableSpring=1, hertz=4.0, dampingRatio=0.5))


def _compare(gpu_lib, build, substeps, frames, small=False):
    from forge2d_gb300.world import GpuWorld
    from oracle.oracle import PortWorld
    wd = scenes.world_def(enableSleep=0)
    if small:
        os.environ["F2D_NO_CLUSTER_SOLVER"] = "1"
    try:
        g = GpuWorld(wd)
    finally:
        os.environ.pop("F2D_NO_CLUSTER_SOLVER", None)
    p = PortWorld(wd)
    for b in (g, p):
        build(b)
    for frame in range(frames):
        g.step(1.0 / 60.0, substeps)
        p.step(1.0 / 60.0, substeps)
        assert g.sync() == 0
        x, y = g.bodies()[:, :9], p.bodies()[:, :9]
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), (frame, np.argwhere(x != y)[:4].tolist())
    overflow = g.counters()["overflow"]
    g.close()
    p.close()
    return overflow


@pytest.mark.parametrize("small", [False, True], ids=["auto", "small"])
@pytest.mark.parametrize("head", ["corner", "middle"])
@pytest.mark.parametrize("count", [266, 267, 268, 700, 1035, 1036, 4000])
def test_contacts_of_one_body(gpu_lib, count, head, small):
    assert _compare(gpu_lib, lambda b: shelves(b, count, head=head), 4, 3, small) == count - 11


def test_contacts_of_a_kinematic_body_in_several_launches(gpu_lib):
    assert _compare(gpu_lib, lambda b: shelves(b, 1500, scenes.KINEMATIC), 10, 2) == 1489


@pytest.mark.parametrize("count", [267, 268, 600])
def test_joints_of_one_body(gpu_lib, count):
    _compare(gpu_lib, lambda b: spokes(b, count), 4, 4)


def test_racks_beside_each_other(gpu_lib):
    """Several such bodies in one world, with contacts and joints on one of them."""
    def build(b):
        shelves(b, 400)
        shelves(b, 300, head="middle", per=60)
        spokes(b, 300)
    _compare(gpu_lib, build, 4, 3)


def test_a_wait_as_long_as_the_chain(gpu_lib):
    """Circles that touch each other wait in their colours for the whole chain
    of a body under 210 thousand of them, some 170 milliseconds in each stage.
    (They come in seven frames: a body's new contacts are coloured one by one,
    100 thousand at most.)"""
    from forge2d_gb300.world import GpuWorld
    from oracle.oracle import PortWorld
    wd = scenes.world_def(enableSleep=0, gravityY=-1.0)
    g, p = GpuWorld(wd), PortWorld(wd)
    for b in (g, p):
        rack = b.create_body(scenes.body_def(type=scenes.KINEMATIC))
        for r in list(range(1, 400)) + [0]:
            b.create_box(rack, scenes.shape_def(), 158.0, 0.1, 158.0, 2.0 * r, 1.0, 0.0)
    for frame in range(7):
        for b in (g, p):
            for k in range(30_000 * frame, 30_000 * frame + 30_000):
                c = b.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=0.26 + 0.52 * (k % 600), positionY=2.0 * (k // 600) + 0.34))
                b.create_circle(c, scenes.shape_def(), 0.0, 0.0, 0.25)
            b.step(1.0 / 60.0, 1)
        assert g.sync() == 0, frame
    x, y = g.bodies()[:, :9], p.bodies()[:, :9]
    assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), np.argwhere(x != y)[:4].tolist()
    assert g.counters()["overflow"] == 210_000 - 11
    g.close()
    p.close()
