"""Tiles of packed points (over 4,096 candidates a search block, over 1,024
pairs a point) against the oracle, bit for bit, in scenes that have enough of
them for a warp each in both passes (the density walk of FL_PASSES_CELL_TASKS,
and the per-point mode's), and in scenes that have few, at the smallest and
the largest density block (one warp that evaluates and adds; thirty-two). How
many tiles fall in each class is counted on the CPU and asserted, so a case
cannot miss the path that it is here for. Bit-equality needs no tolerance.
"""
from __future__ import annotations

import ctypes as C
import functools

import numpy as np
import pytest

import fluids3_gb300 as F
from fluids3_gb300 import scenes
from oracle import oracle as O

from helpers import assert_bit_equal

pytestmark = pytest.mark.gpu
LO, HI = (-60.0, 0.0, -60.0), (60.0, 120.0, 60.0)
UNDEF = 0xFFFFFFFF


def sms() -> int:
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def params():
    return scenes.make_params(LO, HI)


def clusters(p, many, size, few, few_size, thin, seed):
    """`many` clusters of 2 x size points, half of them on either side of a
    face between two cells in x (so a tile holds points of both, and the second
    cell's search block both halves), `few` of few_size points, `thin` points
    anywhere and three outside the grid; all of a cluster within h."""
    rng = np.random.default_rng(seed)
    h = p.psmoothradius / p.sim_scale
    edge = 1.0 / np.array([p.gridDelta[k] for k in range(3)])
    lo = np.array([p.gridMin[k] for k in range(3)])
    at = [(x, y, z) for y in range(2, 22, 3) for z in range(2, 22, 3) for x in range(2, 20, 4)]
    at = [at[k] for k in rng.permutation(len(at))]
    parts = []
    for k, n in enumerate([2 * size] * many + [few_size] * few):
        c = lo + (np.array(at[k]) + (0.0, 0.5, 0.5)) * edge
        d = rng.uniform(0.02, 0.19, (n, 3)) * h * rng.choice([-1.0, 1.0], (n, 3))
        d[:, 0] = np.abs(d[:, 0]) * np.where(np.arange(n) < n // 2, -1.0, 1.0)
        parts.append(c + d)
    parts.append(rng.uniform(np.array(LO) + 3, np.array(HI) - 3, (thin, 3)))
    pos = np.concatenate(parts)
    pos = pos[rng.permutation(len(pos))].astype(np.float32)
    pos[[5, 500, len(pos) - 1]] = [(900.0, 1.0, 1.0), (np.nan, 0.0, 0.0), (1.0, -700.0, 1.0)]
    vel = rng.normal(0, 0.3, pos.shape).astype(np.float32)
    return pos, vel, np.arange(len(pos), dtype=np.uint32)


def classes(p, st):
    """Tiles of the sorted state: crowded, packed in the density pass (by the
    larger search block of its first and last points), packed in the force
    pass (a point of 1,024 pairs)."""
    n = len(st.gcell)
    tiles = -(-n // 32)
    off = st.off.astype(np.int64)
    adj = [(y * p.gridRes[2] + z) * p.gridRes[0] for y in (-1, 0) for z in (-1, 0)]
    inr = np.flatnonzero(st.gcell != UNDEF)
    block = np.zeros(n, np.int64)
    cell = st.gcell[inr].astype(np.int64)
    for a in adj:
        block[inr] += off[cell + a + 1] - off[cell + a - 1]
    last = inr[-1]
    ends = [np.arange(0, last + 1, 32), np.minimum(np.arange(0, last + 1, 32) + 31, last)]
    m = np.maximum(block[ends[0]], block[ends[1]])
    pairs = np.zeros(n + 1, np.uint32)
    O._adj_lib().orc_pairs(C.byref(p), n, *[O._p(a) for a in (st.pos, st.gcell, st.off, st.cnt, pairs)], None)
    own = np.diff(pairs.astype(np.int64))
    most = np.pad(own, (0, tiles * 32 - n)).reshape(tiles, 32).max(1)
    return int(((m >= 1024) & (m < 4096)).sum()), int((m >= 4096).sum()), int((most >= 1024).sum())


@functools.lru_cache(maxsize=None)
def scene(kind):
    p = params()
    if kind == "many":     # a warp per packed tile in the density pass (18 a multiprocessor) and the force pass (32)
        pos, vel, clr = clusters(p, 1024 * sms() // 8600 + 3, 4300, 3, 1100, 4001, 2)
    elif kind == "few":
        pos, vel, clr = clusters(p, 2, 4300, 5, 1250, 3002, 3)
    else:
        pos, vel, clr = clusters(p, 0, 0, 0, 0, 2500, 4)
    sort = O.State.new(p, pos, vel, vel, clr)
    O.insert(p, sort); O.prefix_sum(p, sort); O.counting_sort(p, sort)
    counts = classes(p, sort)
    O.density(p, sort, threads=8); O.force(p, sort, threads=8)
    step = O.State.new(p, pos, vel, vel, clr)
    O.step(p, step, 0.0, threads=8)
    return p, pos, vel, clr, counts, sort, step


def check(kinds, mode, block):
    parts = [scene(k) for k in kinds]
    n = [len(q[1]) for q in parts]
    cat = [np.concatenate([q[k] for q in parts]) for k in (1, 2, 3)]
    s = (F.FluidSystem(parts[0][0], n[0]) if len(parts) == 1 else F.FluidSystem.batch([q[0] for q in parts], n))
    with s:
        s.SetNeighbourPasses(mode)
        s.SetLaunchShapes(density=block)
        s.SetParticles(cat[0], cat[1], cat[1], clr=cat[2])
        s.InsertParticlesCUDA(); s.PrefixSumCellsCUDA(); s.CountingSortFullCUDA()
        s.ComputePressureCUDA(); s.ComputeForceCUDA()
        s.Sync()
        phases = s.state()
        s.ComputePressureCUDA()   # (the tile lists are used up: every tile by its own warp)
        s.Sync()
        again = s.GetBuffer(F.FPRESS)
        s.SetParticles(cat[0], cat[1], cat[1], clr=cat[2])
        s.Run()
        s.Sync()
        fused = s.state()
    base = 0
    for q, m in zip(parts, n):
        at = slice(base, base + m)
        for k in ("clr", "press", "force"):
            assert_bit_equal(phases[k][at], getattr(q[5], k), f"{kinds} {mode} {block}: phases, {k}")
        assert_bit_equal(again[at], q[5].press, f"{kinds} {mode} {block}: density again")
        for k in ("clr", "press", "pos", "vel", "veval"):
            assert_bit_equal(fused[k][at], getattr(q[6], k), f"{kinds} {mode} {block}: fused, {k}")
        base += m


@pytest.mark.parametrize("mode", ["points", "cells"])
@pytest.mark.parametrize("kinds", [("many",), ("thin", "many", "few")])
def test_packed_tiles_for_every_warp_equal_the_oracle(kinds, mode):
    crowded, packed, force = scene("many")[4]
    assert packed >= 18 * sms() and 5 * packed >= 2 * crowded, "the density pass walks them apart"
    assert force >= 32 * sms(), "the force pass gives them a warp each"
    check(kinds, mode, 0)


@pytest.mark.parametrize("block", [32, 1024])
@pytest.mark.parametrize("kinds", [("few",), ("thin", "few")])
def test_a_few_packed_and_crowded_tiles_at_either_end_of_the_blocks(kinds, block):
    crowded, packed, _ = scene("few")[4]
    assert 0 < crowded < 18 * sms() and 0 < packed < 18 * sms(), "both are shared by blocks"
    check(kinds, "cells", block)


@pytest.mark.parametrize("mode", ["cells", "auto"])
def test_replayed_steps_of_packed_scenes_equal_the_per_point_mode(mode):
    p, pos, vel, clr = scene("many")[:4]
    out = {}
    for m in ("points", mode):
        with F.FluidSystem(p, len(pos)) as s:
            s.SetNeighbourPasses(m)
            s.SetParticles(pos, vel, vel, clr=clr)
            s.RunSteps(2)
            s.Sync()
            assert s.NeighbourPassesInUse() == ("points" if m == "points" else "cells")
            s.RunSteps(3)
            s.Sync()
            out[m] = s.state()
    for k in ("clr", "press", "force", "pos", "vel", "veval", "gcell"):
        assert_bit_equal(out[mode][k], out["points"][k], f"{mode}: {k}")
