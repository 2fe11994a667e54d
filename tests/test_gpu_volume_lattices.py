"""Volume sampling against the oracle over both ways and every number of lanes
a voxel: lattices of 20,000 voxels and more, close together (by bricks: ragged,
mostly empty, backwards, out of the grid, long in one axis so that a brick spans
over 32 rows of cells) and far apart, and smaller ones down to a voxel; both
search blocks, and a grid whose points have moved since its sort. The tolerance
is that of the voxel sums elsewhere: they differ from the oracle's through expf,
the rounding of its argument and the order of a sum of positive terms, a few
1e-7 of each."""
from __future__ import annotations

import numpy as np
import pytest

import fluids3_gb300 as F
from fluids3_gb300 import scenes
from oracle import oracle as O

pytestmark = pytest.mark.gpu

RTOL = 1e-5
LO, HI = (-30.0, 0.0, -30.0), (30.0, 60.0, 30.0)
BRICKS = [((33, 29, 23), (-28, 1, -29), (-16, 12, -20)), ((30, 27, 29), (-12, 5, 11), (-28, 1, -9)),
          ((61, 67, 65), LO, HI), ((65, 62, 63), (-50, -15, -45), (10, 35, 10)), ((40, 5, 111), (-26, 0, -28), (-22, 60, -17))]
WIDE = [((64, 64, 65), (-300, -200, -300), (300, 400, 300)), ((80, 80, 50), (-200, -100, -200), (150, 200, 180)),
        ((40, 50, 40), LO, HI), ((32, 32, 32), LO, HI), ((16, 31, 30), LO, HI), ((15, 16, 16), LO, HI), ((7, 1, 3), LO, HI),
        ((1, 1, 1), (-28, 2, -28), (-27, 3, -27))]


@pytest.mark.parametrize("grid_density", [0.75, 2.0])
@pytest.mark.parametrize("moved", [False, True])
def test_every_lattice_equals_the_oracle(grid_density, moved):
    sc = scenes.dam_break(n=9000, seed=5)
    p = scenes.make_params(LO, HI, grid_density=grid_density)
    with F.FluidSystem(p, sc.n) as s:
        s.SetParticles(sc.pos, sc.vel, sc.veval, clr=sc.clr)
        s.RunSteps(3)
        if not moved:
            s.SampleParticles((2, 2, 2), LO, HI)            # bins and sorts
        pos, off, cnt = s.GetBuffer(F.FPOS), s.GetBuffer(F.FGRIDOFF), s.GetBuffer(F.FGRIDCNT)
        for res, lo, hi in BRICKS + WIDE:
            got = s.SampleParticles(res, lo, hi, 0.5, sort_first=False)
            want = O.sample_volume(p, pos, off, cnt, res, np.array(lo, np.float32), np.array(hi, np.float32), 0.5)
            scale = max(float(np.abs(want).max()), 1e-30)
            assert got.shape == want.shape
            assert np.allclose(got, want, rtol=RTOL, atol=RTOL * scale), (res, float(np.abs(got - want).max() / scale))
            assert (want > 0).any() or np.prod(res) < 100


def test_a_volume_without_points_is_zero():
    p = scenes.make_params(LO, HI)
    pos = np.array([[29.0, 59.0, 29.0]], np.float32)
    with F.FluidSystem(p, 1) as s:
        s.SetParticles(pos)
        for res in ((40, 40, 40), (8, 8, 8)):
            assert not s.SampleParticles(res, LO, (10.0, 30.0, 10.0), 1.0).any()


@pytest.mark.parametrize("grid_density", [0.75, 2.0])
@pytest.mark.parametrize("n", [1, 60, 690])
def test_lattices_of_a_mostly_empty_box_equal_the_oracle(n, grid_density):
    """Points whose supports fill little of the box (690: a twentieth of it,
    about), most bricks without one: the lattice of bricks and its neighbours
    in size and spacing."""
    p = scenes.make_params(LO, HI, grid_density=grid_density)
    rng = np.random.default_rng(n)
    pos = (np.array([-12.0, 20.0, 7.0]) + rng.normal(0, 3.0, (n, 3))).astype(np.float32)
    pos[: n // 3] = rng.uniform(np.array(LO) + 2, np.array(HI) - 2, (n // 3, 3))
    with F.FluidSystem(p, n) as s:
        s.SetParticles(pos)
        s.SampleParticles((2, 2, 2), LO, HI)
        got_pos, off, cnt = s.GetBuffer(F.FPOS), s.GetBuffer(F.FGRIDOFF), s.GetBuffer(F.FGRIDCNT)
        for res, lo, hi in (((141, 139, 143), LO, HI), ((61, 67, 65), LO, HI), ((131, 30, 120), (-35, 10, -10), (20, 25, 31))):
            got = s.SampleParticles(res, lo, hi, 0.5, sort_first=False)
            want = O.sample_volume(p, got_pos, off, cnt, res, np.array(lo, np.float32), np.array(hi, np.float32), 0.5)
            scale = max(float(np.abs(want).max()), 1e-30)
            assert np.allclose(got, want, rtol=RTOL, atol=RTOL * scale), (res, float(np.abs(got - want).max() / scale))
            assert (want > 0).any()
