# SPDX-License-Identifier: MIT
"""The work a user of this framework has it do, as measurable cases.

Each case is one pass through the public entry points -- ``pmb200.core.World``
(the tick), ``pmb200.pm.RigidSession`` (the pm* command API) and the C entry
``pmb_mesh_bvh_build`` -- over the framework's own workloads: the cube
pyramid, box piles up to the 65,536-box benchmark pile, joint chains and rigs,
concave meshes, batches of independent scenes, and the learned warm start with
its online training. A tick case advances its world, as a simulation does, and
hands the caller the new states; the roll-out case restores a snapshot first,
as a planner or a learner that replays one state does.
"""
import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "parallel-mater_b200"))
from pmb200 import core, pm, scenes  # noqa: E402

SETTLED = os.path.join(ROOT, "tests", "golden", "settled_pile_64x32x32.npz")
PILE65K = (64, 32, 32)


def listed():
    return [
        # The smallest interactive scene: a game or a robot cell ticks one
        # pyramid of 55 cubes and reads the poses back (launch latency).
        {"name": "pyramid 55, legacy", "kind": "pyramid", "levels": 10, "realtime": False},
        # The same scene through the reference's command API (record, submit,
        # wait, mapped read-back), realtime profile: what a switched-over
        # application runs.
        {"name": "pyramid 55, pm* API", "kind": "driver", "levels": 10},
        # Every joint type in small rigs (a robotics test bench).
        {"name": "joint rigs, 8 scenes", "kind": "rigs", "scenes": 8},
        # Concave and high-triangle meshes: the triangle-mesh narrowphase.
        {"name": "concave meshes, 64 scenes", "kind": "meshes", "scenes": 64},
        # An ordinary box pile, as it lands, at the profile's 10 sweeps.
        {"name": "pile 4096, legacy", "kind": "pile", "gx": 16, "gy": 16, "gz": 16, "realtime": False},
        # A ragged, smaller pile at the realtime profile's 8 sweeps.
        {"name": "pile 1001, realtime", "kind": "pile", "gx": 11, "gy": 7, "gz": 13, "realtime": True},
        # Long joint chains: 33k bodies held by point joints, 20 sweeps.
        {"name": "chains 512x64", "kind": "chains", "count": 512, "links": 64},
        # The benchmark pile in real time: 65,536 boxes, 8 sweeps, stepped
        # and read back every tick.
        {"name": "pile 65536, realtime", "kind": "settled", "realtime": True},
        # The benchmark pile to an equal residual (99.9th percentile within
        # 0.1 mm, at most 64 sweeps), rolled out from one snapshot.
        {"name": "pile 65536, to residual", "kind": "settled", "realtime": False},
        # Many independent scenes stepped as one world (training
        # environments), two ticks per CUDA-graph replay.
        {"name": "batch of 128 scenes", "kind": "batch", "scenes": 128},
        # The learned warm start, trained online while it is used.
        {"name": "pile 4096, learned", "kind": "learned", "gx": 16, "gy": 16, "gz": 16},
        # Mesh upload: the BVH of a large triangle mesh, built on the GPU.
        {"name": "mesh BVH 200k", "kind": "bvh", "triangles": 200_000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pyramid", "driver", "rigs", "meshes", "pile", "pile", "pile", "chains", "batch", "learned",
                       "bvh"])
    if kind == "pyramid":
        return {"kind": kind, "levels": rng.randint(2, 40), "realtime": rng.random() < 0.5}
    if kind == "driver":
        return {"kind": kind, "levels": rng.randint(2, 20)}
    if kind == "rigs":
        return {"kind": kind, "scenes": _log_int(rng, 2, 64)}
    if kind == "meshes":
        return {"kind": kind, "scenes": _log_int(rng, 2, 256)}
    if kind in ("pile", "learned"):
        side = _log_int(rng, 3, 24)
        case = {"kind": kind, "gx": side, "gy": rng.randint(2, 24), "gz": max(2, side + rng.randint(-3, 3))}
        if kind == "pile":
            case["realtime"] = rng.random() < 0.5
        return case
    if kind == "chains":
        return {"kind": kind, "count": _log_int(rng, 1, 512), "links": _log_int(rng, 4, 64)}
    if kind == "batch":
        return {"kind": kind, "scenes": _log_int(rng, 4, 128)}
    return {"kind": "bvh", "triangles": _log_int(rng, 1_000, 200_000)}


# ---------------------------------------------------------------- inputs
def _rng(seed):
    return np.random.Generator(np.random.Philox(seed))


@functools.lru_cache(maxsize=1)
def _settled():
    """The benchmark pile with its committed settled states."""
    s = scenes.box_pile(PILE65K, seed=4)
    z = np.load(SETTLED)
    s.states = np.ascontiguousarray(z["states"], np.float32).view(scenes.STATE_DTYPE).reshape(-1)
    return s


@functools.lru_cache(maxsize=4)
def _batch(count):
    """A mix of `count` independent scenes: box piles and joint chains."""
    return scenes.batched_scenes(count, seed=5)


def _nudged(scene, seed, speed):
    """The scene with seeded velocities added to its dynamic bodies."""
    import dataclasses
    st = scene.states.copy()
    dyn = scene.bodies["motion"] == scenes.DYNAMIC
    r = _rng(seed)
    n = int(dyn.sum())
    st["v"][dyn] += r.uniform(-speed, speed, (n, 3)).astype(np.float32)
    st["w"][dyn] += r.uniform(-speed, speed, (n, 3)).astype(np.float32)
    return dataclasses.replace(scene, states=st)


def _pile_warmup(case):
    # The spawn grid's layers reach the ground and meet: 1.8 m apart, about
    # 40 ticks for the first layer and a few more for each one above.
    return 40 + 3 * case["gy"]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "bvh":
        return _prepare_bvh(case["triangles"], seed)
    if kind == "driver":
        scene = pm.canonical_scene(scenes.pyramid(case["levels"], seed=seed, profile=scenes.REALTIME))
        session = pm.RigidSession(scene, iterations=8, contact_capacity=64 * scene.n + 4096)
        for _ in range(8):
            pm.check(session.step(), "step")
        return {"kind": kind, "session": session}
    replay = restore = False
    learned = None
    contacts = 0  # the default contact capacity
    if kind == "pyramid":
        scene = scenes.pyramid(case["levels"], seed=seed)
        desc = scene.step_desc(profile=scenes.REALTIME if case["realtime"] else scenes.LEGACY)
        warm = 8
    elif kind == "rigs":
        scene = scenes.batch([scenes.joint_zoo(seed=1000 * seed + k) for k in range(case["scenes"])], "rigs")
        desc, warm = scene.step_desc(), 8
    elif kind == "meshes":
        scene = scenes.batch([scenes.mesh_mix(seed=1000 * seed + k, margin=0.04 if k % 2 else 0.005)
                              for k in range(case["scenes"])], "meshes")
        desc, warm = scene.step_desc(), 40
        contacts = 1024 * scene.n  # the mesh path's triangle pairs count against it (about 300 a body)
    elif kind == "pile":
        scene = scenes.box_pile((case["gx"], case["gy"], case["gz"]), seed=seed)
        desc = scene.step_desc(profile=scenes.REALTIME if case["realtime"] else scenes.LEGACY)
        warm = _pile_warmup(case)
    elif kind == "learned":
        scene = scenes.box_pile((case["gx"], case["gy"], case["gz"]), seed=seed)
        desc = scene.step_desc(warm_start=1)
        warm, learned = _pile_warmup(case), {"lr": 1e-3, "steps_per_tick": 2}
    elif kind == "chains":
        scene = scenes.chains(case["count"], case["links"], seed=seed)
        desc, warm = scene.step_desc(), 8
    elif kind == "batch":
        scene = _nudged(_batch(case["scenes"]), seed, 0.05)
        desc, warm, replay = scene.step_desc(), 60, True
    elif kind == "settled":
        scene = _nudged(_settled(), seed, 0.01)
        if case["realtime"]:
            desc = scene.step_desc(profile=scenes.REALTIME)
        else:
            desc = scene.step_desc(residual_tolerance=1e-4, max_iterations=64, residual_norm=2)
            restore = True
        warm = 6
    else:
        raise ValueError(kind)
    world = core.World(scene, contact_capacity=contacts)
    if learned:
        world.mlp_attach(seed=1)
        world.mlp_train(True, **learned)
    for _ in range(warm):
        world.step(desc, stats=False)
    if restore:
        world.snapshot()
    if replay:
        world.capture(2, desc)
    return {"kind": kind, "world": world, "desc": desc, "restore": restore, "replay": replay,
            "learned": learned is not None}


def _prepare_bvh(triangles, seed):
    """A rough closed-ish sheet of `triangles` triangles with a random
    storage order, vertices and indices on the device."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    side = max(1, int(math.ceil(math.sqrt(triangles / 2))))
    xs = torch.arange(side + 1, device="cuda", dtype=torch.float32) / side
    x, z = torch.meshgrid(xs, xs, indexing="ij")
    y = 0.2 * torch.sin(9.0 * x) * torch.cos(7.0 * z)
    v = torch.stack([x, y, z], -1).reshape(-1, 3)
    v = (v + torch.rand(v.shape, generator=g, device="cuda") * (0.3 / side)).contiguous()
    k = torch.arange(side * side, device="cuda")
    a = k // side * (side + 1) + k % side
    tri = torch.stack([torch.stack([a, a + 1, a + side + 1], -1),
                       torch.stack([a + 1, a + side + 2, a + side + 1], -1)], 1).reshape(-1, 3)
    tri = tri[torch.randperm(len(tri), generator=g, device="cuda")[:triangles]]
    idx = tri.to(torch.int32).contiguous()
    return {"kind": "bvh", "v": v, "idx": idx,
            "order": torch.zeros(triangles, dtype=torch.int32, device="cuda"),
            "nodes": torch.zeros((2 * triangles, 10), dtype=torch.int32, device="cuda"),
            "count": ctypes.c_uint32()}


# ---------------------------------------------------------------- one pass
def _numbers(states):
    return np.ascontiguousarray(states).view(np.float32).reshape(-1, 13)


def _stats(s):
    return {"whole": np.array([int(s[k]) for k in ("candidate_pairs", "active_pairs", "contacts", "colors", "islands",
                                                   "iterations", "impact", "status")]),
            "residual": np.array([s["residual"], s["residual_max"], s["residual_over"]], np.float32)}


def run(state):
    kind = state["kind"]
    if kind == "bvh":
        rc = core.lib().pmb_mesh_bvh_build(
            state["v"].data_ptr(), len(state["v"]), state["idx"].data_ptr(), state["idx"].numel(),
            state["order"].data_ptr(), state["nodes"].data_ptr(), len(state["nodes"]), ctypes.byref(state["count"]),
            torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        nodes = state["nodes"][:state["count"].value]
        return {"order": state["order"], "bounds": nodes[:, :6].view(torch.float32), "links": nodes[:, 6:]}
    if kind == "driver":
        pm.check(state["session"].step(), "step")
        return _numbers(state["session"].states())
    world = state["world"]
    if state["replay"]:
        world.replay()
        return {"states": _numbers(world.states())}
    if state["restore"]:
        world.restore()
    stats = world.step(state["desc"])
    out = {"states": _numbers(world.states()), **_stats(stats)}
    if state["learned"]:
        out["params"] = world.mlp_params()[0]
    return out


# ---------------------------------------------------------------- its floor
def _shape(case):
    """(bodies, joints, contact points, sweeps, ticks) of one pass: contact
    points per body as these scenes have them at rest or in motion."""
    kind = case["kind"]
    if kind in ("pyramid", "driver"):
        n = case["levels"] * (case["levels"] + 1) // 2
        sweeps = 8 if kind == "driver" or case["realtime"] else 10
        return n, 0, 8 * n, sweeps, 1
    if kind == "rigs":
        return 28 * case["scenes"], 17 * case["scenes"], 0, 12, 1
    if kind == "meshes":
        return 8 * case["scenes"], 0, 24 * case["scenes"], 10, 1
    if kind in ("pile", "learned"):
        n = case["gx"] * case["gy"] * case["gz"]
        return n, 0, 3 * n, 8 if case.get("realtime") else 10, 1
    if kind == "chains":
        n = case["count"] * (case["links"] + 2)
        return n, case["count"] * (case["links"] + 1), 0, 20, 1
    if kind == "settled":
        n = PILE65K[0] * PILE65K[1] * PILE65K[2]
        return n, 0, int(6.6 * n), 8 if case["realtime"] else 50, 1
    sizes, piles = scenes.batched_plan(case["scenes"], 5)
    n = int(sizes.sum())
    chained = int(sizes[~piles].sum())
    return n, chained, 4 * (n - chained), 15, 2


def work(case):
    if case["kind"] == "bvh":
        t = case["triangles"]
        # vertices (half a vertex per triangle) and indices in, order and
        # nodes (about half a node per triangle) out
        return {"bytes": t * (6 + 12 + 4 + 20), "flops": t * 12 * max(1.0, math.log2(t / 4.0))}
    n, joints, contacts, sweeps, ticks = _shape(case)
    # Per tick: a body's state in and out (52 B each), its parameters (52 B)
    # and its mesh (a box: 8 vertices, 12 triangles with planes, about 400 B);
    # a contact's cached record in and out (7 x 16 B each); a joint's record
    # (220 B) and its rows (3 of 88 B) in and out. The states also go to the
    # caller's memory (52 B per body).
    byte = ticks * (n * (3 * 52 + 400) + contacts * 224 + joints * (220 + 2 * 264)) + 52 * n
    # Per sweep: a contact's three rows into two 6x6 blocks (27 entries x 3
    # operations x 3 rows x 2 bodies), its errors and projection, its dual
    # update (about 700 in all); a joint's rows likewise; a body's LDL^T
    # solve (about 250).
    flops = ticks * sweeps * (contacts * 700 + joints * 900 + n * 250)
    if case["kind"] == "learned":
        # inference and two training steps (3 x forward) of 8-64-64-2
        flops += contacts * (1 + 2 * 3) * 2 * (8 * 64 + 64 * 64 + 64 * 2)
    return {"bytes": byte, "flops": flops}


def tolerance(case):
    if case["kind"] == "bvh":
        return "exact"  # an order, links, and bounds copied from the vertices
    if case["kind"] == "learned":
        # The predictor's products are bf16 with 32-bit sums; gradients summed
        # in another order move a parameter by a few 1e-4 of its Adam step,
        # and the tick follows the predicted warm start.
        return {"rel": 2e-3, "max": 0.1}
    # The tick's contract is the reference's operation order, bit for bit
    # (states equal the serial restatement's bits); only the residual's RMS is
    # a sum whose order is free, 64-bit sums rounded to 32 bits.
    return {"rel": 5e-7, "max": 5e-6}


def exact(case, seed):
    """None: a tick is a serial Gauss-Seidel sweep over clipped manifolds, and
    its warm contact cache needs tens of earlier ticks; in plain 64-bit numpy
    that takes minutes, and a 64-bit trajectory leaves the 32-bit one at the
    first landing impact (millimetres within 30 ticks)."""
    return None
