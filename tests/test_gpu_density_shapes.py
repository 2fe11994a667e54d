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


@pytest.mark.parametrize("cells,runs", [(1, 1), (6, 1), (7, 1), (4, 4), (5, 5), (6, 2), (7, 2), (32, 1)])
@pytest.mark.parametrize("batch", [False, True])
def test_warps_of_as_many_cells_and_runs_as_share_a_walk_and_one_more(cells, runs, batch):
    """32 points in `cells` cells of one row, `runs` runs of them three cells
    apart, with their neighbours in the rows below: alone in their scene, so
    that they are one warp's."""
    p = scenes.make_params((0.0, 0.0, 0.0), (250.0, 60.0, 60.0))
    rng = np.random.default_rng(cells * 8 + runs)
    edge = 1.0 / np.array([p.gridDelta[k] for k in range(3)])
    xs = [c + 4 * (c * runs // cells) for c in range(cells)]
    at = np.array([(4 + xs[k * cells // 32], 5, 5) for k in range(32)], float)
    pos = np.array([p.gridMin[k] for k in range(3)]) + (at + rng.uniform(0.01, 0.99, (32, 3))) * edge
    below = pos[rng.integers(0, 32, 300)] - rng.uniform(0.0, 0.9, (300, 3)) * edge * (0.5, 1.0, 1.0)
    below[:, 1] = np.minimum(below[:, 1], p.gridMin[1] + 4.999 * edge[1])
    pos = np.concatenate([below, pos]).astype(np.float32)   # (the lower rows of cells sort first)
    pad = 32 - len(below) % 32
    pos = np.concatenate([pos[:pad], pos])[: len(pos) + pad]
    pos[:pad, 1] = p.gridMin[1] + 1.5 * edge[1]
    vel = rng.normal(0, 0.3, pos.shape).astype(np.float32)
    ref = O.State.new(p, pos, vel, vel)
    O.insert(p, ref); O.prefix_sum(p, ref); O.counting_sort(p, ref)
    row = ref.gcell[-32:].astype(np.int64)
    assert len(ref.gcell) % 32 == 0 and len(np.unique(row)) == cells and (np.diff(np.unique(row)) > 2).sum() == runs - 1
    O.density(p, ref); O.force(p, ref)
    n = len(pos)
    k = 2 if batch else 1
    with (F.FluidSystem.batch([p, p], [n, n]) if batch else F.FluidSystem(p, n)) as s:
        s.SetParticles(np.concatenate([pos] * k), np.concatenate([vel] * k), np.concatenate([vel] * k))
        s.InsertParticlesCUDA(); s.PrefixSumCellsCUDA(); s.CountingSortFullCUDA()
        s.ComputePressureCUDA(); s.ComputeForceCUDA()
        s.Sync()
        got = s.state()
    for j in range(k):
        for f in ("pos", "press", "force"):
            assert_bit_equal(got[f][j * n:(j + 1) * n], getattr(ref, f), f"{cells} cells, {runs} runs: {f}")
