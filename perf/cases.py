"""The work that a user of the GPU world has it do, as measurable cases.

A pass is one frame of a program that uses the library: the frame's input
(mouse targets, destroyed and created bodies), one world step, the events,
transforms and query answers that such a program reads. The scenes are those
of ``forge2d_gb300.scenes``, at sizes from a small game scene to the 100k
pile; every pass goes through the C ABI (``include/forge2d_gb300.h``), results
are read into host buffers that the program keeps. One case is the learned
warm start's network: the gradient of a training step and a prediction.

``prepare`` builds the scene (a level's load) and steps it ``frames`` times, so
that passes start from a world whose bodies lie on each other.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from forge2d_gb300 import native, scenes
from forge2d_gb300.world import GpuWorld, WarmStartModel

DT = 1.0 / 60.0

# the full-size mixed pile: 100k bodies over a 400 x 800 spawn region; smaller
# piles keep its density and aspect
PILE_FULL = 100_000


def listed():
    return [
        # a small game scene, every frame: motors, a cart, lifts and three bodies dragged by the mouse; sleeping on
        # (forge2d's default). Launch count and latency are all there is.
        dict(name="rigs", kind="rigs", copies=3, frames=60),
        # the 820-box pyramid with a ball thrown at it: the plain solver-bound stack of one screen
        dict(name="pyramid", kind="pyramids", pyramids=1, rows=40, chains=0, links=0, frames=40),
        # sensor zones over a heap whose bodies they report, begin and end events read
        dict(name="sensors", kind="sensors", count=2000, frames=160),
        # a heap that a program follows by contact events: begin, end and hit events read every frame
        dict(name="pile_events", kind="pile", count=3001, frames=200, sleep=False, events=True),
        # one-sided chain terrain with convex and concave vertices under a heap of mixed shapes
        dict(name="terrain", kind="terrain", count=6007, frames=240),
        # the quarter-size mixed pile
        dict(name="pile_25k", kind="pile", count=25_000, frames=400, sleep=False, events=False),
        # a running game over a big heap, sleeping on: bodies destroyed and created, the step, move events read for
        # the renderer, rays and box queries answered
        dict(name="game_20k", kind="game", count=20_000, spawn=16, rays=16, boxes=4, frames=300),
        # 64 pyramids and 200 revolute chains: stacking plus 10k joints
        dict(name="pyramids_chains", kind="pyramids", pyramids=64, rows=40, chains=200, links=50, frames=60),
        # a large pile with sleeping on (islands kept every step), awake: it is still falling
        dict(name="pile_sleep_60k", kind="pile", count=60_001, frames=300, sleep=True, events=False),
        # many small independent worlds in one step (a training or tuning program's batch)
        dict(name="batched_512", kind="batched", worlds=512, layout=7, frames=120),
        # the headline workload: the 100k mixed pile, dense
        dict(name="pile_100k", kind="pile", count=PILE_FULL, frames=500, sleep=False, events=False),
        # one gradient of the learned warm start's training and a prediction of as many rows
        dict(name="learned_64k", kind="learned", rows=65_536),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rigs", "pyramids", "sensors", "pile", "pile", "pile", "terrain", "game", "batched", "learned"])
    if kind == "rigs":
        return dict(kind=kind, copies=_log_int(rng, 1, 64), frames=rng.randint(20, 90))
    if kind == "pyramids":
        return dict(kind=kind, pyramids=_log_int(rng, 1, 40), rows=rng.randint(8, 40), chains=rng.randint(0, 100),
                    links=rng.randint(5, 50), frames=rng.randint(20, 60))
    if kind == "sensors":
        return dict(kind=kind, count=_log_int(rng, 100, 8000), frames=rng.randint(60, 200))
    if kind == "pile":
        return dict(kind=kind, count=_log_int(rng, 200, 80_000), frames=rng.randint(150, 400),
                    sleep=rng.random() < 0.5, events=rng.random() < 0.4)
    if kind == "terrain":
        return dict(kind=kind, count=_log_int(rng, 200, 20_000), frames=rng.randint(100, 300))
    if kind == "game":
        return dict(kind=kind, count=_log_int(rng, 500, 30_000), spawn=rng.randint(1, 32), rays=rng.randint(1, 32),
                    boxes=rng.randint(1, 8), frames=rng.randint(100, 300))
    if kind == "batched":
        return dict(kind=kind, worlds=_log_int(rng, 8, 400), layout=rng.randint(1, 1 << 20), frames=rng.randint(60, 160))
    return dict(kind=kind, rows=_log_int(rng, 500, 200_000))


# ---------------------------------------------------------------------------
# worlds
# ---------------------------------------------------------------------------
class _Loader(GpuWorld):
    """GpuWorld whose creation calls refill one definition struct, as a
    program that loads a level does; the definitions it is given are whole."""

    def __init__(self, world_def):
        super().__init__(world_def)
        self._bd, self._sdef = native.BodyDef(), native.ShapeDef()
        self._bdp, self._sdp = C.byref(self._bd), C.byref(self._sdef)
        self._i1, self._g = C.c_int32(0), C.c_int32(0)
        self._i1p, self._gp = C.byref(self._i1), C.byref(self._g)

    def create_body(self, body_def):
        s = self._bd
        for k, v in body_def.items():
            setattr(s, k, v)
        if not self.lib.f2d_create_body(self.id, self._bdp, self._i1p, self._gp):
            raise RuntimeError("createBody failed")
        h = (self._i1.value, self._g.value)
        self._wg["body"][h[0] - 1] = h[1]
        return h

    def _sd(self, sd):
        s = self._sdef
        for k, v in sd.items():
            setattr(s, k, v)
        return self._sdp


def _ptr(t, kind):
    return C.cast(t.data_ptr(), C.POINTER(kind))


def _pinned(rows, cols, dtype):
    return torch.zeros((max(rows, 1), cols), dtype=dtype, pin_memory=True)


class _Frame:
    """A world and the host buffers of the program that steps it."""

    LOADER = _Loader

    def __init__(self, world_def):
        self.w = self.LOADER(world_def)
        self.lib, self.id = self.w.lib, self.w.id

    def settle(self, frames):
        for _ in range(frames):
            self.step()
        self.n = self.lib.f2d_world_body_capacity(self.id)
        self.rows = _pinned(self.n, 12, torch.float32)
        self.rows_p = _ptr(self.rows, C.c_float)
        if self.w.sync():
            raise RuntimeError("step status")

    def step(self):
        self.lib.f2d_world_step(self.id, DT, 4)

    def bodies(self):
        self.lib.f2d_world_get_bodies(self.id, self.rows_p, self.n)
        return self.rows

    def one_pass(self):
        self.step()
        return {"bodies": self.bodies()}


class _Rigs(_Frame):
    def __init__(self, case, seed):
        super().__init__(scenes.world_def())
        rng = np.random.default_rng(seed)
        self.mice = scenes.joint_rigs(self.w, copies=case["copies"])
        self.phase = float(rng.uniform(0.0, 2.0 * math.pi))
        self.centres = [(-30.0 * case["copies"] + 25.0 + 30.0 * k + float(rng.uniform(-0.5, 0.5)), 3.0)
                        for k in range(case["copies"])]
        self.settle(case["frames"])

    def step(self):
        self.phase += 0.05
        dx, dy = 1.5 * math.cos(self.phase), 1.0 * math.sin(self.phase)
        for j, (x, y) in zip(self.mice, self.centres):
            self.lib.f2d_mouse_joint_set_target(j[0], j[1], x + dx, y + dy)
        super().step()


class _Pyramids(_Frame):
    def __init__(self, case, seed):
        super().__init__(scenes.world_def(enableSleep=0))
        rng = np.random.default_rng(seed)
        p, rows = case["pyramids"], case["rows"]
        scenes.pyramids_chains(self.w, pyramids=p, rows=rows, chains=case["chains"], links=case["links"])
        pitch = rows + 2.0
        for k in range(p):
            x = -0.5 * p * pitch + (k + 0.5) * pitch
            b = self.w.create_body(scenes.body_def(type=scenes.DYNAMIC, positionX=x + float(rng.uniform(-0.3, 0.3)) * rows,
                                                   positionY=rows + 6.0 + float(rng.uniform(0.0, 6.0)),
                                                   linearVelocityX=float(rng.uniform(-4.0, 4.0)),
                                                   linearVelocityY=float(rng.uniform(-12.0, -2.0))))
            self.w.create_circle(b, scenes.shape_def(density=2.0), 0.0, 0.0, float(rng.uniform(0.5, 1.0)))
        self.settle(case["frames"])


class _Pile(_Frame):
    CAP = 1 << 14

    def __init__(self, case, seed):
        super().__init__(scenes.world_def(enableSleep=int(case["sleep"])))
        scale = math.sqrt(case["count"] / PILE_FULL)
        ev = bool(case["events"])
        scenes.pile(self.w, count=case["count"], seed=seed, width=400.0 * scale, height=800.0 * scale,
                    enable_hit_events=ev, enable_contact_events=ev)
        self.events = ev
        if ev:
            self.b4 = torch.zeros((self.CAP, 4), dtype=torch.int32)
            self.e4 = torch.zeros((self.CAP, 4), dtype=torch.int32)
            self.h4 = torch.zeros((self.CAP, 4), dtype=torch.int32)
            self.h5 = torch.zeros((self.CAP, 5), dtype=torch.float32)
            self.b4_p, self.e4_p, self.h4_p = (_ptr(t, C.c_int32) for t in (self.b4, self.e4, self.h4))
            self.h5_p = _ptr(self.h5, C.c_float)
        self.settle(case["frames"])

    def one_pass(self):
        out = super().one_pass()
        if self.events:
            lib = self.lib
            nb = lib.f2d_world_get_begin_events(self.id, self.b4_p, self.CAP)
            ne = lib.f2d_world_get_end_events(self.id, self.e4_p, self.CAP)
            nh = lib.f2d_world_get_hit_events(self.id, self.h4_p, self.h5_p, self.CAP)
            # hit events come in no set order: a program whose runs repeat sorts them by their shapes
            h4, h5 = self.h4[:nh].numpy(), self.h5[:nh].numpy()
            by = np.lexsort((h4[:, 2], h4[:, 0]))
            h4[:], h5[:] = h4[by], h5[by]
            out.update(counts=np.array([nb, ne, nh], np.int32), begin=self.b4, end=self.e4, hit=self.h4, hit_at=self.h5)
        return out


class _Sensors(_Frame):
    CAP = 1 << 14

    def __init__(self, case, seed):
        super().__init__(scenes.world_def(enableSleep=0))
        scale = math.sqrt(case["count"] / 300.0)
        scenes.sensor_field(self.w, count=case["count"], seed=seed, width=30.0 * scale, height=40.0 * scale)
        self.b4 = torch.zeros((self.CAP, 4), dtype=torch.int32)
        self.e4 = torch.zeros((self.CAP, 4), dtype=torch.int32)
        self.settle(case["frames"])

    def one_pass(self):
        out = super().one_pass()
        ne = C.c_int32(0)
        nb = self.lib.f2d_world_get_sensor_events(self.id, _ptr(self.b4, C.c_int32), _ptr(self.e4, C.c_int32), self.CAP,
                                                  C.byref(ne))
        out.update(counts=np.array([nb, ne.value], np.int32), begin=self.b4, end=self.e4)
        return out


class _Terrain(_Frame):
    def __init__(self, case, seed):
        super().__init__(scenes.world_def(enableSleep=0))
        scale = math.sqrt(case["count"] / 400.0)
        scenes.chain_terrain(self.w, count=case["count"], seed=seed, width=40.0 * scale, height=40.0 * scale,
                             bumps=max(1, round(6.0 * scale)))
        self.settle(case["frames"])


class _Turned(_Loader):
    """Loader that turns each sub-world's gravity by an angle of the seed."""

    def turn(self, seed):
        self.turns = np.random.default_rng(seed)

    def begin_subworld(self, gx, gy):
        a = float(self.turns.uniform(-0.1, 0.1))
        c, s = math.cos(a), math.sin(a)
        return super().begin_subworld(c * gx - s * gy, s * gx + c * gy)


class _Batched(_Frame):
    """The sub-worlds' sizes are the layout's; the seed turns their gravity."""

    LOADER = _Turned

    def __init__(self, case, seed):
        super().__init__(scenes.world_def(enableSleep=0))
        self.w.turn(seed)
        scenes.batched(self.w, worlds=case["worlds"], seed=case["layout"])
        self.settle(case["frames"])


class _Game(_Frame):
    """Each pass: the oldest ``spawn`` bodies are destroyed and as many thrown
    in from above, the world steps, the renderer reads the move events, and
    ``rays`` closest rays and ``boxes`` box queries are answered."""

    def __init__(self, case, seed):
        super().__init__(scenes.world_def(enableSleep=1))
        scale = math.sqrt(case["count"] / PILE_FULL)
        self.half, self.top = 200.0 * scale, 800.0 * scale
        self.alive = list(scenes.pile(self.w, count=case["count"], seed=seed, width=2.0 * self.half, height=self.top))
        self.rng = np.random.default_rng(seed + 1)
        self.spawn, self.rays, self.boxes = case["spawn"], case["rays"], case["boxes"]
        self.oldest = 0
        self.body, self.shape = scenes.body_def(type=scenes.DYNAMIC), scenes.shape_def()
        cap = 1 << 12
        self.cap = cap
        self.ray_shape = torch.zeros((self.rays, 2), dtype=torch.int32)
        self.ray_out = torch.zeros((self.rays, 5), dtype=torch.float32)
        self.box_out = torch.zeros((self.boxes, cap, 2), dtype=torch.int32)
        self.ray_p = [(_ptr(self.ray_shape[k], C.c_int32), _ptr(self.ray_out[k], C.c_float)) for k in range(self.rays)]
        self.box_p = [_ptr(self.box_out[k], C.c_int32) for k in range(self.boxes)]
        self.settle(case["frames"])
        self.moved_i, self.moved_f = _pinned(self.n, 3, torch.int32), _pinned(self.n, 4, torch.float32)
        self.moved_p = (_ptr(self.moved_i, C.c_int32), _ptr(self.moved_f, C.c_float))

    def one_pass(self):
        w, lib = self.w, self.lib
        x = self.rng.uniform(-self.half + 1.0, self.half - 1.0, self.spawn)
        y = self.rng.uniform(0.8 * self.top, self.top, self.spawn)
        for k in range(self.spawn):
            at = self.oldest % len(self.alive)
            w.destroy_body(self.alive[at])
            self.body["positionX"], self.body["positionY"] = float(x[k]), float(y[k])
            b = w.create_body(self.body)
            w.create_circle(b, self.shape, 0.0, 0.0, 0.5)
            self.alive[at] = b
            self.oldest += 1
        self.step()
        n = lib.f2d_world_get_body_events(self.id, *self.moved_p, self.n)
        q = self.rng.uniform(-1.0, 1.0, (self.rays + self.boxes, 4))
        hit = []
        self.ray_shape.zero_()
        self.ray_out.zero_()
        for k in range(self.rays):
            ox, oy, tx, ty = (float(v) for v in q[k])
            hit.append(lib.f2d_world_cast_ray_closest(self.id, ox * self.half, (0.5 + 0.5 * oy) * self.top, tx * self.half,
                                                      ty * 0.5 * self.top, 1, -1, *self.ray_p[k]))
        counts = []
        for k in range(self.boxes):
            cx, cy = float(q[self.rays + k, 0]) * self.half, (0.25 + 0.25 * float(q[self.rays + k, 1])) * self.top
            r = 3.0 + 2.0 * float(q[self.rays + k, 2])
            counts.append(lib.f2d_world_overlap_aabb(self.id, cx - r, cy - r, cx + r, cy + r, 1, -1, self.box_p[k], self.cap))
        return {"counts": np.array([n] + hit + counts, np.int32), "moved": self.moved_i, "moved_to": self.moved_f,
                "ray_shape": self.ray_shape, "ray": self.ray_out, "boxes": self.box_out}


# ---------------------------------------------------------------------------
# the learned warm start's network
# ---------------------------------------------------------------------------
def _learned_inputs(case, seed):
    """Feature and target rows as the solver records them for new contact
    points: unit normal, relative velocity, separation, anchors, inverse
    masses, friction; the two impulses a step ended with."""
    rng = np.random.default_rng(seed)
    n = case["rows"]
    a = rng.uniform(-math.pi, math.pi, n)
    s = np.zeros((n, 14), np.float32)
    s[:, 0], s[:, 1] = np.cos(a), np.sin(a)
    s[:, 2:4] = rng.normal(0.0, 2.0, (n, 2))
    s[:, 4] = rng.uniform(-0.02, 0.02, n)
    s[:, 5:9] = rng.uniform(-0.8, 0.8, (n, 4))
    s[:, 9:11] = rng.lognormal(0.3, 0.5, (n, 2))
    s[:, 11] = rng.choice([0.3, 0.6, 0.9], n)
    push = np.maximum(0.0, -s[:, 3]) + 0.1 * rng.exponential(1.0, n)
    s[:, 12] = push / s[:, 9]
    s[:, 13] = np.clip(-0.4 * s[:, 2], -0.6, 0.6) * s[:, 12]
    mean = s.mean(0, dtype=np.float64)
    std = s.std(0, dtype=np.float64)
    return s, mean.astype(np.float32), (1.0 / std).astype(np.float32)


_W = (("W1", 64, 16), ("W2", 64, 64), ("W3", 8, 64))


def _learned_params(seed):
    """Weights of the network's scale in the order of f2d_mlp_get_params."""
    rng = np.random.default_rng(seed + 77)
    w1 = np.zeros((64, 16), np.float32)
    w1[:, :12] = rng.uniform(-1.0, 1.0, (64, 12)) * math.sqrt(6.0 / 12.0)
    w2 = (rng.uniform(-1.0, 1.0, (64, 64)) * math.sqrt(6.0 / 64.0)).astype(np.float32)
    w3 = np.zeros((8, 64), np.float32)
    w3[:2] = rng.uniform(-1.0, 1.0, (2, 64)) * math.sqrt(6.0 / 64.0)
    b1, b2, b3 = (rng.normal(0.0, 0.05, k).astype(np.float32) for k in (64, 64, 8))
    b3[2:] = 0.0
    return w1, w2, w3, b1, b2, b3


class _Learned:
    def __init__(self, case, seed):
        self.s, mean, inv = _learned_inputs(case, seed)
        self.feats = np.ascontiguousarray(self.s[:, :12])
        self.model = WarmStartModel(seed=1)
        self.model.set_normalization(mean, inv)
        self.model.set_params(np.concatenate([p.reshape(-1) for p in _learned_params(seed)]))

    def one_pass(self):
        grad, loss = self.model.gradient(self.s)
        return {"grad": grad, "loss": float(loss), "predicted": self.model.predict(self.feats)}


def exact(case, seed):
    """The network's gradient, loss and predictions in 64 bits. A world step
    has no such value: a pass continues from the state its 32-bit steps made."""
    if case["kind"] != "learned":
        return None
    s, mean, inv = _learned_inputs(case, seed)
    w1, w2, w3, b1, b2, b3 = (torch.from_numpy(p).double() for p in _learned_params(seed))
    for p in (w1, w2, w3, b1, b2, b3):
        p.requires_grad_(True)
    z = (torch.from_numpy(s).double() - torch.from_numpy(mean).double()) * torch.from_numpy(inv).double()
    x = torch.nn.functional.pad(z[:, :12], (0, 4))
    h = torch.relu(torch.relu(x @ w1.T + b1) @ w2.T + b2)
    y = (h @ w3.T + b3)[:, :2]
    loss = 0.5 * (y - z[:, 12:]).square().sum() / len(s)
    loss.backward()
    pred = y.detach() / torch.from_numpy(inv[12:]).double() + torch.from_numpy(mean[12:]).double()
    return {"grad": torch.cat([p.grad.reshape(-1) for p in (w1, w2, w3, b1, b2, b3)]), "loss": float(loss.detach()),
            "predicted": pred}


# ---------------------------------------------------------------------------
_KINDS = {"rigs": _Rigs, "pyramids": _Pyramids, "pile": _Pile, "sensors": _Sensors, "terrain": _Terrain,
          "batched": _Batched, "game": _Game, "learned": _Learned}


def prepare(case, seed):
    return _KINDS[case["kind"]](case, seed)


def run(state):
    return state.one_pass()


def _counts(case):
    """(bodies, touching contacts, joints) of the case's scene, about."""
    k = case["kind"]
    if k == "rigs":
        return 12 * case["copies"], 8 * case["copies"], 9 * case["copies"]
    if k == "pyramids":
        r, p, links = case["rows"], case["pyramids"], case["chains"] * case["links"]
        return p * (r * (r + 1) // 2 + 1) + links, int(p * 1.45 * r * (r + 1)), links
    if k == "batched":
        # a third each of pyramids (mean 172 boxes), piles (260 shapes) and chains (55 links)
        w = case["worlds"]
        return int(w * 165), int(w * 340), int(w * 18)
    return case["count"], int(2.1 * case["count"]), 0


def work(case):
    """Bytes and operations a pass cannot do without. A step reads and writes
    each body's state once (transform, velocities, sweep: 64 B), reads its
    mass and force rows and its shape's geometry and material (168 B), writes
    its shape's two boxes (32 B) and hands its row to the program (48 B); it
    reads and writes each touching contact's manifold (96 B and 16 B of keys);
    a joint's definition and impulses are read, the impulses written. Per
    contact a step computes a manifold and, in each of 4 substeps, a warm
    start, a solve and a relax of two points: about 4 000 operations."""
    if case["kind"] == "learned":
        n, params = case["rows"], 64 * 16 + 64 * 64 + 8 * 64 + 136
        macs = 12 * 64 + 64 * 64 + 64 * 2
        return {"bytes": n * (14 + 12 + 2) * 4 + params * 8, "flops": 2.0 * n * macs * 4}
    b, c, j = _counts(case)
    return {"bytes": b * (2 * 64 + 168 + 32 + 48) + c * (2 * 96 + 16) + j * (160 + 2 * 24),
            "flops": c * 4000.0 + j * 1500.0 + b * 300.0}
