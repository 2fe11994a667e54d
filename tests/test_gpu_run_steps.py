"""RunSteps (graph-replayed step pairs) around changes of the state it was
captured on, bit-equal to single Run steps of a fresh system. Bit-equality
needs no tolerance.
"""
from __future__ import annotations

import time

import numpy as np
import pytest

import fluids3_gb300 as F
from fluids3_gb300 import scenes

from helpers import FIELDS, assert_bit_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first,more", [(2000, 1000), (100, 100), (2048, 1)])
def test_restoring_a_checkpoint_of_fewer_points_steps_those_points(first, more):
    """A checkpoint of `first` points, restored after a RunSteps call on
    `first + more`: the next RunSteps call steps `first` points (and after a
    restore of the larger state, all of them)."""
    sc = scenes.dam_break(n=first + more, seed=19)
    a, b = slice(0, first), slice(first, None)
    want = {}
    for n in (first, first + more):
        with F.FluidSystem(sc.params, n) as s:
            s.SetParticles(sc.pos[:n], sc.vel[:n], sc.veval[:n], clr=sc.clr[:n])
            for _ in range(4):
                s.Run()
            s.Sync()
            want[n] = s.state()
    with F.FluidSystem(sc.params, first + more) as s:
        s.SetParticles(sc.pos[a], sc.vel[a], sc.veval[a], clr=sc.clr[a])
        s.SaveCheckpoint(0)
        s.AddParticles(sc.pos[b], sc.vel[b], sc.veval[b], clr=sc.clr[b])
        s.SaveCheckpoint(1)
        s.RunSteps(4)
        for slot, n in ((0, first), (1, first + more), (0, first)):
            s.RestoreCheckpoint(slot)
            s.RunSteps(4)
            s.Sync()
            assert s.NumPoints() == n
            got = s.state()
            for k in FIELDS + ("gridcnt", "gridoff"):
                assert_bit_equal(got[k], want[n][k], f"{n} points restored: {k}")


@pytest.mark.parametrize("steps", [33, 50, 64])
def test_calls_of_up_to_64_steps_return_before_the_queued_work_is_done(steps):
    """RunSteps queues its steps and returns: behind 64 queued steps, a call
    of 33 to 64 leaves most of that work unfinished when it returns, in the
    default mode as with the per-point passes. (Were it to wait for its first
    steps, the queued ones would be done by then.) The states are equal."""
    sc = scenes.wave_tank(n=1_000_000)
    out = {}
    for mode in ("auto", "points"):
        with F.FluidSystem(sc.params, sc.n) as s:
            s.SetNeighbourPasses(mode)
            s.SetParticles(sc.pos, sc.vel, sc.veval, clr=sc.clr)
            s.RunSteps(2)   # captures the pair
            s.Sync()
            t0 = time.perf_counter()
            s.RunSteps(64)
            s.RunSteps(steps)
            t1 = time.perf_counter()
            s.Sync()
            t2 = time.perf_counter()
            # (waiting for the queued 64 takes a third or more of the time)
            assert t1 - t0 < 0.2 * (t2 - t0), (mode, t1 - t0, t2 - t0)
            assert sum(s.PassesSteps()) == 2 + 64 + steps
            out[mode] = s.state()
    for k in FIELDS + ("gridcnt", "gridoff"):
        assert_bit_equal(out["auto"][k], out["points"][k], f"{steps} steps: {k}")


@pytest.mark.parametrize("keep,want", [(True, (4, 0)), (False, (0, 4))])
def test_what_replayed_steps_of_a_tape_count_as(keep, want):
    """Backward replays the steps of each segment: with kept pair lists they
    count as per-point steps, else by the mode set. (Taped steps count as
    per-point steps in every mode.)"""
    sc = scenes.dam_break(n=3000, seed=5)
    w = np.ones((3, sc.n, 3), np.float32)
    with F.FluidSystem(sc.params, sc.n) as s:
        s.SetParticles(sc.pos, sc.vel, sc.veval, clr=sc.clr)
        s.SetNeighbourPasses("cells")
        s.TapeBegin(4, 2, keep_lists=keep)
        for _ in range(4):
            s.Run()
        assert s.PassesSteps() == (4, 0)
        s.Backward(*w)
        assert tuple(a - b for a, b in zip(s.PassesSteps(), (4, 0))) == want
        assert s.NeighbourPasses() == "cells"
