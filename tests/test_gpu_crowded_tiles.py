"""Crowded tiles of 32 slots against the oracle, bit for bit, on both sides of
the rules that choose who takes them: tiles shared by whole blocks (few of
them), a warp each once there are tiles for every warp (the force pass's
needs about 78,000 points), packed tiles (over 4,096 candidates or 1,024
pairs a point) that fall in a class of their own, tiles of several scenes of
a batch, and, with gridSrch 3, lists that fill at very different rates within
a warp. Phases, two fused steps and a batch. Bit-equality needs no tolerance.
"""
from __future__ import annotations

import numpy as np
import pytest

import fluids3_gb300 as F
from fluids3_gb300 import scenes
from oracle import oracle as O

from helpers import assert_bit_equal

pytestmark = pytest.mark.gpu
LO, HI = (-40.0, 0.0, -40.0), (40.0, 80.0, 40.0)


def ball(rng, n, pairs, h):
    """n points in a ball, about `pairs` within h of each."""
    r = h * (n / pairs) ** (1.0 / 3.0)
    d = rng.normal(size=(n, 3))
    return np.array([0.0, 40.0, 0.0]) + r * rng.random((n, 1)) ** (1 / 3) * d / np.linalg.norm(d, axis=1, keepdims=True)


def cloud(kind, h, seed):
    rng = np.random.default_rng(seed)
    thin = lambda n: rng.uniform(np.asarray(LO) + 2, np.asarray(HI) - 2, (n, 3))
    if kind == "shared":        # a few hundred crowded tiles among thin ones, some packed
        p = np.concatenate([ball(rng, 6000, 400, h), ball(rng, 3000, 2500, h) + 15.0, thin(9000)])
    elif kind == "alone":       # more crowded tiles than warps
        p = ball(rng, 100000, 260, h)
    elif kind == "packed":      # more packed tiles than warps, in a small ball
        p = ball(rng, 100000, 1500, h)
    elif kind == "mixed":       # warps to themselves for the crowded tiles, blocks for the packed
        p = np.concatenate([ball(rng, 92000, 220, h), ball(rng, 5000, 2000, h) + 24.0])
    else:                       # "ramp": density grows along x, lists of few to over a hundred pairs
        n = 3000
        x = 12 * h * rng.random(n) ** 0.35
        p = np.stack([x - 6 * h, 30 + 4 * h * rng.random(n), 4 * h * rng.random(n)], 1)
    return p.astype(np.float32)


def state_of(kind, cell_h, seed):
    p = scenes.make_params(LO, HI, grid_density=1.5 / cell_h)
    pos = cloud(kind, p.psmoothradius / p.sim_scale, seed)
    n = len(pos)
    vel = np.random.default_rng(seed + 1).normal(0, 0.3, (n, 3)).astype(np.float32)
    return p, pos, vel, np.arange(n, dtype=np.uint32)


CASES = [("shared", 2.0), ("alone", 2.0), ("packed", 2.0), ("mixed", 2.0), ("shared", 0.75), ("ramp", 0.75),
         ("ramp", 2.0)]


@pytest.mark.parametrize("kind,cell_h", CASES)
def test_phases_and_fused_steps_equal_the_oracle(kind, cell_h):
    p, pos, vel, clr = state_of(kind, cell_h, 3)
    n = len(pos)
    ref = O.State.new(p, pos, vel, vel, clr)
    O.insert(p, ref); O.prefix_sum(p, ref); O.counting_sort(p, ref)
    O.density(p, ref, threads=8); O.force(p, ref, threads=8)
    with F.FluidSystem(p, n) as s:
        s.SetParticles(pos, vel, vel, clr=clr)
        s.InsertParticlesCUDA(); s.PrefixSumCellsCUDA(); s.CountingSortFullCUDA()
        s.ComputePressureCUDA(); s.ComputeForceCUDA()
        s.Sync()
        got = s.state()
        for k in ("clr", "press", "force"):
            assert_bit_equal(got[k], getattr(ref, k), f"{kind} {cell_h}: phases, {k}")
    ref = O.State.new(p, pos, vel, vel, clr)
    with F.FluidSystem(p, n) as s:
        s.SetParticles(pos, vel, vel, clr=clr)
        for _ in range(2):
            O.step(p, ref, s.time, threads=8)
            s.Run()
        s.Sync()
        got = s.state()
    for k in ("clr", "press", "pos", "vel", "veval"):
        assert_bit_equal(got[k], getattr(ref, k), f"{kind} {cell_h}: fused, {k}")


@pytest.mark.parametrize("kinds", [("shared", "ramp", "shared"), ("mixed", "shared", "ramp")])
@pytest.mark.parametrize("cell_h", [2.0, 0.75])
def test_batched_scenes_equal_the_oracle(kinds, cell_h):
    parts = [state_of(k, cell_h, 11 + i) for i, k in enumerate(kinds)]
    with F.FluidSystem.batch([q[0] for q in parts], [len(q[1]) for q in parts]) as b:
        cat = [np.concatenate([q[k] for q in parts]) for k in (1, 2, 3)]
        b.SetParticles(cat[0], cat[1], cat[1], clr=cat[2])
        b.Run()
        b.Sync()
        got = b.state()
        infos = [b.SceneInfo(k) for k in range(len(parts))]
    for (p, pos, vel, clr), info, kind in zip(parts, infos, kinds):
        ref = O.State.new(p, pos, vel, vel, clr)
        O.step(p, ref, 0.0, threads=8)
        a, n = info["point_base"], info["n"]
        for k in ("clr", "press", "pos", "vel"):
            assert_bit_equal(got[k][a:a + n], getattr(ref, k), f"{kind} {cell_h}: batch, {k}")
