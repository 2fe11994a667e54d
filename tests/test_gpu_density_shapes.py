"""The density pass at every pinned block size: the block that SetLaunchShapes
accepts is the one that runs (with gridSrch 3 and for positions that have
moved since the sort as with gridSrch 2), and densities, pair counts (through
the forces) and order equal the oracle's bit for bit. Bit-equality needs no
tolerance.
"""
from __future__ import annotations

import numpy as np
import pytest

import fluids3_gb300 as F
from fluids3_gb300 import scenes
from oracle import oracle as O

from helpers import assert_bit_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cell_h", [0.75, 2.0])   # gridSrch 3, 2
@pytest.mark.parametrize("block", [0, 32, 96, 256, 288, 512, 1024])
@pytest.mark.parametrize("batch", [False, True])
def test_a_pinned_density_block_is_the_one_that_runs(cell_h, block, batch):
    sc = scenes.dam_break(n=5000, seed=17)   # (rows of up to 1024 threads, the last block ragged)
    p = scenes.make_params(sc.params.bound_min, sc.params.bound_max, grid_density=1.5 / cell_h)
    ref = O.State.new(p, sc.pos, sc.vel, sc.veval, sc.clr)
    O.insert(p, ref); O.prefix_sum(p, ref); O.counting_sort(p, ref)
    O.density(p, ref, threads=8); O.force(p, ref, threads=8)
    s = F.FluidSystem.batch([p, p], [sc.n, sc.n]) if batch else F.FluidSystem(p, sc.n)
    with s:
        s.SetLaunchShapes(density=block)
        k = 2 if batch else 1
        s.SetParticles(*[np.concatenate([v] * k) for v in (sc.pos, sc.vel, sc.veval)], clr=np.concatenate([sc.clr] * k))
        s.InsertParticlesCUDA(); s.PrefixSumCellsCUDA(); s.CountingSortFullCUDA()
        s.ComputePressureCUDA(); s.ComputeForceCUDA()
        s.Sync()
        assert F.lib().fl_test_density_block(s.handle) == (block or s.LaunchShapes()["density"])
        got = s.state()
        for j in range(k):
            for f in ("clr", "press", "force"):
                assert_bit_equal(got[f][j * sc.n:(j + 1) * sc.n], getattr(ref, f), f"{cell_h} {block} {j}: {f}")
        # positions that have moved since the sort go by the rows whatever gridSrch is
        s.AdvanceCUDA(0.0, 0.0, p.sim_scale)   # (dt 0: they keep their values)
        s.ComputePressureCUDA()
        s.Sync()
        assert F.lib().fl_test_density_block(s.handle) == (block or s.LaunchShapes()["density"])
        moved = s.GetBuffer(F.FPRESS)
        for j in range(k):
            assert_bit_equal(moved[j * sc.n:(j + 1) * sc.n], ref.press, f"{cell_h} {block} {j}: density again")
