"""RunSteps (graph-replayed step pairs) around changes of the state it was
captured on, bit-equal to single Run steps of a fresh system. Bit-equality
needs no tolerance.
"""
from __future__ import annotations

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
