"""Volume sampling by bricks and by wide voxels against the oracle: lattices
that do not divide into bricks, voxels from a fraction of h to many cells
apart, boxes that reach out of the grid or run backwards, the 3 x 3 x 3 search
block, and a grid whose points have moved since its sort. The tolerance is
that of the voxel sums elsewhere: they differ from the oracle's through expf
and the rounding of its argument, a few 1e-7 of each (positive) term."""
from __future__ import annotations

import numpy as np
import pytest

import fluids3_gb300 as F
from fluids3_gb300 import scenes
from oracle import oracle as O

pytestmark = pytest.mark.gpu

RTOL = 1e-5
LO, HI = (-30.0, 0.0, -30.0), (30.0, 60.0, 30.0)


def close(got, want, what):
    scale = max(float(np.abs(want).max()), 1e-30)
    assert np.allclose(got, want, rtol=RTOL, atol=RTOL * scale), (what, float(np.abs(got - want).max() / scale))


@pytest.mark.parametrize("grid_density", [0.75, 2.0])
@pytest.mark.parametrize("moved", [False, True])
def test_volume_equals_the_oracle(grid_density, moved):
    sc = scenes.dam_break(n=9000, seed=5)
    p = scenes.make_params(LO, HI, grid_density=grid_density)
    boxes = [((33, 17, 9), LO, HI), ((1, 2, 3), LO, HI), ((6, 5, 4), LO, HI), ((31, 3, 40), (-28, 2, -29), (-12, 9, 11)),
             ((20, 20, 20), (-55, -20, -50), (10, 30, 15)), ((9, 30, 10), (-20, 20, 5), (-28, 3, -25))]
    with F.FluidSystem(p, sc.n) as s:
        s.SetParticles(sc.pos, sc.vel, sc.veval, clr=sc.clr)
        s.RunSteps(3)
        if not moved:
            s.SampleParticles((2, 2, 2), LO, HI)            # bins and sorts
        pos, off, cnt = s.GetBuffer(F.FPOS), s.GetBuffer(F.FGRIDOFF), s.GetBuffer(F.FGRIDCNT)
        for res, lo, hi in boxes:
            got = s.SampleParticles(res, lo, hi, 0.5, sort_first=False)
            want = O.sample_volume(p, pos, off, cnt, res, np.array(lo, np.float32), np.array(hi, np.float32), 0.5)
            close(got, want, (res, lo, hi))
            assert (want > 0).any() or res == (1, 2, 3)
