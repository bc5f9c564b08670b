# SPDX-License-Identifier: MIT
"""The tick's size-dependent branches at their edges, against the oracle.

A tick picks kernels and grids by the world's size: one solve block up to 40
bodies, narrowphase lanes up to 6,144, a one-block grid up to 8,192 buckets
(4,096 bodies), a one-block colour order up to 8,192 bodies; a query keeps 64 candidates; a lane group takes two, five or ten joints
of a body at a time. Every branch evaluates the serial order's operations, so states,
candidate pairs and colours are compared bit for bit.
"""
import ctypes
import re

import numpy as np
import pytest

import oracle as O
from pmb200 import core, scenes

pytestmark = pytest.mark.gpu


def _same(scene, ticks, contact_capacity=0, **kw):
    w, o = core.World(scene, contact_capacity=contact_capacity), O.OracleWorld(scene)
    contacts = 0
    for t in range(ticks):
        sg, so = w.step(**kw), o.step(**kw)
        assert sg["status"] == 0, core.status_names(int(sg["status"]))
        for k in ("candidate_pairs", "active_pairs", "contacts", "colors", "islands"):
            assert sg[k] == so[k], (t, k)
        assert np.array_equal(w.candidate_pairs(), o.candidate_pairs()), t
        dyn = scene.bodies["motion"] == scenes.DYNAMIC
        assert np.array_equal(w.graph()[0][dyn], o.graph()[0][dyn]), t
        assert np.array_equal(w.states().view(np.uint8), o.states().view(np.uint8)), t
        contacts = max(contacts, int(sg["contacts"]))
    w.close()
    return contacts


# box_pile adds five static bodies; boxes 1.4 m apart touch from the start.
@pytest.mark.parametrize("bodies", [6, 40, 41, 130, 1030, 4096, 4097, 6144, 6145, 8192, 8193])
def test_world_sizes_around_the_dispatch_edges(gpu_available, bodies):
    side = max(1, int(np.ceil((bodies - 5) ** (1.0 / 3.0))))
    scene = scenes.box_pile((side, side, side), seed=bodies, spacing=1.4, count=bodies - 5)
    assert scene.n == bodies
    assert _same(scene, 6 if bodies < 2000 else 2) > 0 or bodies < 10


def test_query_with_more_candidates_than_are_kept(gpu_available):
    """A plate over 12 x 12 boxes (144 candidates) and boxes below the kept
    number, in one world."""
    b = scenes._Builder()
    scenes._ground(b, 20.0, 20.0)
    cube = b.mesh(*scenes.box_mesh((0.25, 0.25, 0.25)))
    plate = b.mesh(*scenes.box_mesh((4.0, 0.1, 4.0)))
    b.body(plate, scenes.DYNAMIC, (0.0, 0.62, 0.0), mass=5.0, inertia=scenes.box_inertia(5.0, (4.0, 0.1, 4.0)))
    for k in range(144):
        x, z = (k % 12 - 5.5) * 0.6, (k // 12 - 5.5) * 0.6
        b.body(cube, scenes.DYNAMIC, (x, 0.2505, z), mass=1.0, inertia=scenes.box_inertia(1.0, (0.25,) * 3))
    assert _same(b.build("plate", 10), 4) > 0


def _plate_scene():
    """A plate over 12 x 12 boxes, and the boxes on the ground: one query of
    145 candidates and 144 of a few."""
    b = scenes._Builder()
    scenes._ground(b, 20.0, 20.0)
    cube = b.mesh(*scenes.box_mesh((0.25, 0.25, 0.25)))
    plate = b.mesh(*scenes.box_mesh((4.0, 0.1, 4.0)))
    for k in range(144):
        x, z = (k % 12 - 5.5) * 0.55, (k // 12 - 5.5) * 0.55
        b.body(cube, scenes.DYNAMIC, (x, 0.2505, z), mass=1.0, inertia=scenes.box_inertia(1.0, (0.25,) * 3))
        if k == 71:
            b.body(plate, scenes.DYNAMIC, (0.0, 0.62, 0.0), mass=5.0, inertia=scenes.box_inertia(5.0, (4.0, 0.1, 4.0)))
    return b.build("plate between", 10)


@pytest.mark.parametrize("past", [1, 70])
def test_a_query_cut_off_by_the_candidate_capacity(gpu_available, past):
    """The capacity ends inside a body's segment (`past` candidates into it; 70
    are past the kept ones): the tick reports the overflow, keeps as many
    candidates as fit, in order and out of the full set, and goes on."""
    scene = _plate_scene()
    o = O.OracleWorld(scene)
    o.step()
    full = o.candidate_pairs()
    query = full // scene.n
    first, many = np.unique(query, return_index=True)[1], np.unique(query, return_counts=True)[1]
    at = int(np.nonzero(many > past + 1)[0][-1])
    capacity = int(first[at]) + past
    assert many[at] > past and capacity < len(full)
    w = core.World(scene, candidate_capacity=capacity)
    for t in range(3):
        st = w.step()
        assert int(st["status"]) & 1, core.status_names(int(st["status"]))
        assert st["candidate_pairs"] == capacity
        codes = w.candidate_pairs()
        assert len(codes) == capacity and (codes // scene.n < scene.n).all()
        assert (np.diff(codes.astype(np.int64)) > 0).all()  # by query body, then by identity
        if t == 0:
            assert np.array_equal(codes[:first[at]], full[:first[at]])  # the whole segments before it
            assert np.isin(codes[first[at]:], full[first[at]:first[at] + many[at]]).all()
        assert np.isfinite(w.states()["x"]).all()
    w.close()


def _cone(sides, radius, height):
    """A cone of `sides` faces, its base (y = 0) triangulated as a fan."""
    a = 2.0 * np.pi * np.arange(sides) / sides
    v = np.stack([radius * np.cos(a), np.zeros(sides), radius * np.sin(a)], -1)
    v = np.concatenate([v, [[0.0, height, 0.0]]]).astype(np.float32)
    t = [(k, (k + 1) % sides, sides) for k in range(sides)] + [(0, k, k + 1) for k in range(1, sides - 1)]
    return v, scenes._fix_winding(v, np.array(t, np.uint32))


@pytest.mark.parametrize("speed", [0.0, 9.0])
def test_polygons_that_outgrow_the_lanes(gpu_available, speed):
    """Cones of 32 triangles, the face path's most: a 17-sided base within one
    triangle of a plate's top clips that triangle to 17 vertices, one more than
    a pair's lanes hold. The plates come first, so at equal separations the
    cone's base is the reference face. Resting, and falling past the margin
    without turning (a swept pair)."""
    sides = 17
    v, t = _cone(sides, 1.0, 1.5)
    assert len(t) == 96
    b = scenes._Builder()
    scenes._ground(b, 100.0, 100.0)
    plate = b.mesh(*scenes.box_mesh((4.0, 0.25, 4.0)))
    cone = b.mesh(v, t)
    spots = [(12.0 * (k % 4), 12.0 * (k // 4)) for k in range(16)]
    for x, z in spots:
        b.body(plate, scenes.DYNAMIC, (x, 0.25, z), mass=200.0, inertia=scenes.box_inertia(200.0, (4.0, 0.25, 4.0)))
    rng = np.random.Generator(np.random.Philox(5))
    for k, (x, z) in enumerate(spots):
        turn = float(rng.uniform(-3, 3))
        side = 2.0 if k % 2 else -2.0  # either triangle of the plate's top
        b.body(cone, scenes.DYNAMIC, (x + side, 0.5 + 0.09 * (speed > 0), z + side),
               q=(0.0, float(np.sin(turn / 2)), 0.0, float(np.cos(turn / 2))), v=(0.0, -speed, 0.0), mass=2.0,
               inertia=(0.5, 0.5, 0.5))
    scene = b.build("cones", 10)
    assert _same(scene, 6, contact_capacity=1 << 18) > 0


@pytest.mark.parametrize("joints", [1, 2, 3, 5, 6, 11, 23])
def test_bodies_with_many_joints(gpu_available, joints):
    """A hub joined to `joints` boxes by joints of every type in turn (generic
    and spring joints have more rows an axis than a lane's slot holds)."""
    b = scenes._Builder()
    hub = b.mesh(*scenes.box_mesh((0.3, 0.3, 0.3)))
    small = b.mesh(*scenes.box_mesh((0.05, 0.05, 0.05)))
    h = b.body(hub, scenes.DYNAMIC, (0.0, 3.0, 0.0), w=(0.3, 0.5, -0.2), mass=4.0,
               inertia=scenes.box_inertia(4.0, (0.3,) * 3))
    rng = np.random.Generator(np.random.Philox(joints))
    for k in range(joints):
        a = 2.0 * np.pi * k / joints
        x = np.array([np.cos(a), 0.2 * (k % 3), np.sin(a)])
        v = tuple(float(q) for q in rng.uniform(-1, 1, 3))
        i = b.body(small, scenes.DYNAMIC, tuple(float(q) for q in x + (0.0, 3.0, 0.0)), v=v, mass=0.5,
                   inertia=scenes.box_inertia(0.5, (0.05,) * 3))
        j = b.joint(k % 8, h, i, tuple(float(q) for q in 0.5 * x), tuple(float(q) for q in -0.5 * x))
        o = b.joints[j]
        o["lin_limit_axes"] = o["ang_limit_axes"] = 7
        o["lin_lower"], o["lin_upper"] = (-0.1, -0.1, 0.0), (0.2, 0.1, 0.0)
        o["ang_lower"], o["ang_upper"] = (-0.3, -0.2, -0.4), (0.3, 0.2, 0.4)
        o["lin_spring_axes"] = o["ang_spring_axes"] = 7
        o["lin_stiffness"], o["lin_damping"] = (200.0,) * 3, (5.0,) * 3
        o["ang_stiffness"], o["ang_damping"] = (50.0,) * 3, (1.0,) * 3
        o["motor_angular"] = o["motor_linear"] = 1
        o["motor_angular_velocity"], o["motor_angular_max_impulse"] = 2.0, 5.0
        o["motor_linear_velocity"], o["motor_linear_max_impulse"] = 0.5, 3.0
    _same(b.build("hub", 12), 12)


def test_block_solves_over_forty_decades(gpu_available):
    """Random symmetric positive blocks, with zero entries and entries near
    the ends of the 32-bit range: the device's solution is the serial one's
    bit pattern."""
    rng = np.random.Generator(np.random.Philox(12))
    rows = []
    for k in range(20000):
        m = rng.uniform(-1, 1, (6, 6)) * 10.0 ** rng.uniform(-3, 3, (6, 1))
        h = m @ m.T + np.diag(10.0 ** rng.uniform(-4, 2, 6))
        if k % 3 == 0:
            h[3:, :3] = h[:3, 3:] = 0.0
        h = h * 10.0 ** rng.uniform(-20, 15)
        g = rng.uniform(-1, 1, 6) * 10.0 ** rng.uniform(-22, 12)
        if k % 5 == 0:
            g[rng.integers(0, 6, 3)] = -0.0
        rows.append(np.concatenate([[h[r, c] for r in range(6) for c in range(r + 1)], g]))
    x = np.array(rows, np.float32)
    out = core.math_eval(0, x)
    want = [O.block_solve(r[:21], r[21:]) for r in x]
    assert np.array_equal(out[:, 6].astype(bool), np.array([bool(w[0]) for w in want]))
    got, ref = out[:, :6].copy(), np.array([w[1] for w in want], np.float32)
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))
    assert (out[:, 6] == 1).sum() > 15000


def test_a_body_per_thread(gpu_available):
    """Colours with more bodies than a round of 16-lane groups holds give them
    a thread each (policy 4): 21,952 boxes, contacts from the start, the same
    bits as the oracle under every CTA size."""
    scene = scenes.box_pile((28, 28, 28), seed=3, spacing=1.42)
    o = O.OracleWorld(scene)
    want = []
    for _ in range(2):
        o.step(iterations=3)
        want.append(o.states().view(np.uint8).copy())
    for variant in (0, 1, 2):
        w = core.World(scene)
        w.set_launch_plan(variant, 4)
        for t in range(2):
            assert w.step(iterations=3)["status"] == 0
            assert np.array_equal(w.states().view(np.uint8), want[t]), (variant, t)
        w.close()


def test_groups_that_solve_resting_and_flying_bodies_in_turn(gpu_available):
    """A lane group's next body reuses the shared memory its lanes read the
    last one's block from. 12,544 boxes of one colour, half of them in the air
    (no rows: the block is the first thing written) and the others sliding or
    lifting off (crossing rows, two passes), mixed in one sort class: more than
    a round for the groups of every CTA size."""
    b = scenes._Builder()
    side = 112
    scenes._ground(b, 1.5 * side + 5.0, 1.5 * side + 5.0)
    cube = b.mesh(*scenes.box_mesh((0.5, 0.5, 0.5)))
    rng = np.random.Generator(np.random.Philox(8))
    for k in range(side * side):
        x, z = (k % side - 0.5 * side) * 3.0, (k // side - 0.5 * side) * 3.0
        v = rng.uniform(-1, 1, (2, 3))
        b.body(cube, scenes.DYNAMIC, (x, 0.499 if rng.random() < 0.5 else 5.0, z), v=tuple(map(float, v[0])),
               w=tuple(map(float, v[1])), mass=1.0, inertia=scenes.box_inertia(1.0, (0.5,) * 3))
    scene = b.build("resting and flying", 4)
    o = O.OracleWorld(scene)
    want = []
    for _ in range(3):
        o.step()
        want.append(o.states().view(np.uint8).copy())
    for variant in (0, 1, 2):
        w = core.World(scene)
        w.set_launch_plan(variant, 1)
        for t in range(3):
            st = w.step()
            assert st["status"] == 0 and st["colors"] == 1 and st["contacts"] > 10000
            assert np.array_equal(w.states().view(np.uint8), want[t]), (variant, t)
        w.close()


def test_translating_pairs_that_try_several_manifolds(gpu_available):
    """Boxes that move more than their margin without turning: sliding ones
    touch at the start (the predicted poses), rising ones no longer do (the
    start's poses, then the correction's), falling ones touch on the way --
    the polygons of one pair's manifolds share the lanes' shared memory."""
    b = scenes._Builder()
    scenes._ground(b, 60.0, 60.0)
    cube = b.mesh(*scenes.box_mesh((0.5, 0.5, 0.5)))
    rng = np.random.Generator(np.random.Philox(21))
    for k in range(96):
        x, z = (k % 12 - 5.5) * 2.0, (k // 12 - 3.5) * 2.0
        kind = k % 4
        y, v = [(0.5005, (6.0, 0.0, 2.0)), (0.5005, (0.5, 6.0, 0.0)), (1.1, (3.0, -40.0, 1.0)),
                (1.1, (60.0, -20.0, 45.0))][kind]
        v = tuple(float(q) for q in np.array(v) * rng.uniform(0.7, 1.3))
        for up in range(2):
            b.body(cube, scenes.DYNAMIC, (x + 0.1 * up, y + 1.0005 * up, z), v=v, mass=1.0,
                   inertia=scenes.box_inertia(1.0, (0.5,) * 3))
    # Pairs without a face manifold take the triangle path: at most 2 x 12 x 12
    # triangle pairs for each of at most 1,600 candidates.
    assert _same(b.build("translating", 8), 4, contact_capacity=1600 * 288) > 0


class _Telemetry(ctypes.Structure):
    _fields_ = [("tick", ctypes.c_uint64)] + [(k, ctypes.c_uint64 * 7) for k in
                                              ("dispatches", "workgroups", "bytes_moved", "barriers")] + \
               [("sweeps", ctypes.c_uint64), ("spatial_builds", ctypes.c_uint64)]


def _telemetry(w):
    t = _Telemetry()
    f = core.lib().pmb_world_tick_telemetry
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p]
    assert f(w.h, ctypes.byref(t)) == 0
    return t


@pytest.mark.parametrize("profile", [scenes.LEGACY, scenes.REALTIME])
@pytest.mark.parametrize("variant", [0, 3])
@pytest.mark.parametrize("boxes", [20, 2000])
def test_telemetry_counts_the_barriers_a_tick_passes(gpu_available, boxes, variant, profile):
    """One barrier a colour round; in a sweep one a colour and, in the group
    variants, one after the duals. A legacy tick with an impact sweeps twice,
    a realtime tick once."""
    w = core.World(scenes.box_pile((13, 13, 13), seed=5, spacing=1.4, count=boxes))
    w.set_launch_plan(variant, 0)
    for _ in range(4):
        w.step(profile=profile, stats=False)
    report = w.profile_step(profile=profile)
    st, t = w.stats(), _telemetry(w)
    rounds = int(re.search(r"rounds (\d+)", report).group(1))
    sweeps = int(st["iterations"]) * (2 if st["impact"] and profile == scenes.LEGACY else 1)
    assert rounds >= 1 and st["colors"] > 1 and t.sweeps == sweeps > 0
    assert t.barriers[4] == rounds + sweeps * (int(st["colors"]) + (1 if variant < 3 else 0))
    assert sum(t.barriers) == t.barriers[4]
    w.close()


@pytest.mark.parametrize("boxes", [20, 300])
def test_a_barrier_limit_keeps_the_worlds_grid(gpu_available, boxes):
    """A limit that can only run out by a fault leaves the launches and the
    states as they are; one below 1,024 polls takes every block."""
    scene = scenes.box_pile((7, 7, 7), seed=6, spacing=1.4, count=boxes)
    states, groups = [], []
    for limit in (0, 1 << 20):
        w = core.World(scene)
        w.set_barrier_limit(limit)
        for _ in range(3):
            assert w.step()["status"] == 0
        states.append(w.states().view(np.uint8))
        groups.append(list(_telemetry(w).workgroups))
        if limit:
            w.set_barrier_limit(1)
            w.step()
            assert _telemetry(w).workgroups[4] > groups[0][4] + 148
        w.close()
    assert np.array_equal(states[0], states[1]) and groups[0] == groups[1]
