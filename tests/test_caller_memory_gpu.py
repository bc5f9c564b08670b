# SPDX-License-Identifier: MIT
"""Worlds in caller-owned memory whose scratch range does not survive a tick.

Scratch is rebuilt by every tick (pmb_world_memory_requirements), so its owner
may write it between ticks, or hand one range to several worlds that tick in
turn. The states must stay the oracle's, bit for bit.
"""
import ctypes

import numpy as np
import pytest

import oracle as O
from pmb200 import core, scenes

pytestmark = pytest.mark.gpu


def _requirements(scene):
    return core.memory_requirements(scene.n, len(scene.joints), len(scene.mesh_vertex_offsets) - 1,
                                    len(scene.vertices), len(scene.indices) // 3)


class CallerWorld(core.World):
    """A world in the given device ranges (int32 tensors; allocations are
    512-byte aligned)."""

    def __init__(self, scene, persistent, scratch):
        self.scene, s = scene, scene
        self._keep = [np.ascontiguousarray(x) for x in (s.bodies, s.states, s.mesh_vertex_offsets, s.vertices,
                                                         s.mesh_index_offsets, s.indices, s.joints)]
        b, st, vo, v, io, i, j = (k.ctypes.data if k.size else None for k in self._keep)
        d = core.WorldDesc(scene.n, b, st, len(s.mesh_vertex_offsets) - 1, vo, v, io, i, len(s.joints), j)
        d.persistent_memory, d.persistent_bytes = persistent.data_ptr(), 4 * persistent.numel()
        d.scratch_memory, d.scratch_bytes = scratch.data_ptr(), 4 * scratch.numel()
        h = ctypes.c_void_p()
        assert core.lib().pmb_world_create(ctypes.byref(d), ctypes.byref(h)) == 0
        self.h = h


def _words(size):
    import torch
    return torch.zeros((size + 3) // 4, dtype=torch.int32, device="cuda")


def _pile():
    return scenes.box_pile((7, 5, 7), seed=3, spacing=1.4)  # touching from the start


@pytest.mark.parametrize("scene", [_pile, scenes.joint_zoo, scenes.mesh_mix], ids=["no joints", "joints", "meshes"])
def test_scratch_overwritten_between_ticks(gpu_available, scene):
    import torch
    scene = scene()
    persistent, scratch = (_words(size) for size in _requirements(scene))
    # Small and different words: whatever a tick took from them as an offset
    # or an index would give wrong results, but none out of range.
    garbage = torch.arange(scratch.numel(), dtype=torch.int32, device="cuda") % 7 + 1
    torch.cuda.synchronize()
    w, o = CallerWorld(scene, persistent, scratch), O.OracleWorld(scene)
    for t in range(8):
        scratch.copy_(garbage)
        torch.cuda.synchronize()
        assert w.step()["status"] == 0
        o.step()
        assert np.array_equal(w.states().view(np.uint8), o.states().view(np.uint8)), t
    w.close()


def test_worlds_that_share_one_scratch_range(gpu_available):
    """A world with joints and one without, ticked in turn over one range."""
    import torch
    pair = [scenes.joint_zoo(), _pile()]
    sizes = [_requirements(s) for s in pair]
    persistent = [_words(p) for p, _ in sizes]
    scratch = _words(max(s for _, s in sizes))
    torch.cuda.synchronize()
    worlds = [CallerWorld(s, p, scratch) for s, p in zip(pair, persistent)]
    oracles = [O.OracleWorld(s) for s in pair]
    for t in range(8):
        for w, o in zip(worlds, oracles):
            assert w.step()["status"] == 0
            o.step()
            assert np.array_equal(w.states().view(np.uint8), o.states().view(np.uint8)), t
    for w in worlds:
        w.close()
