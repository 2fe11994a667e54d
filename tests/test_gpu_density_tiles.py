"""The density pass's warps of 32 slots against the oracle, bit for bit, where
they can go wrong: sizes around a warp, cells from just over h to many times
h (the filter's units), points spread so thin that a warp holds many runs
of cells, rows of cells that end inside a warp, crowded cells (several rounds
of candidates), points outside the grid, and the per-point rows of
gridSrch > 2. Forces are compared too: they come from the pair lists that
the density pass records. Bit-equality needs no tolerance.
"""
from __future__ import annotations

import numpy as np
import pytest

import fluids3_gb300 as F
from fluids3_gb300 import scenes
from oracle import oracle as O

from helpers import assert_bit_equal

pytestmark = pytest.mark.gpu


def cloud(kind: str, n: int, h: float, lo, hi, seed: int) -> np.ndarray:
    rng = np.random.default_rng(seed)
    lo, hi = np.asarray(lo), np.asarray(hi)
    if kind == "thin":         # many cells between neighbours
        p = rng.uniform(lo + 1, hi - 1, (n, 3))
    elif kind == "dense":      # about 40 points per (2h)^3
        edge = h * (n / 5.0) ** (1.0 / 3.0)
        p = lo + 3 + rng.random((n, 3)) * np.minimum(np.maximum(edge, h), hi - lo - 6)
    elif kind == "clump":      # a ball of radius 0.7 h and a thin rest
        p = rng.uniform(lo + 1, hi - 1, (n, 3))
        m = (2 * n) // 3
        d = rng.normal(size=(m, 3))
        p[:m] = (lo + hi) / 2 + 0.7 * h * rng.random((m, 1)) ** (1 / 3) * d / np.linalg.norm(d, axis=1, keepdims=True)
    else:                      # "column": one cell wide in x, so a row of cells ends every few points
        p = lo + 3 + rng.random((n, 3)) * np.array([1.5 * h, min(12 * h, hi[1] - lo[1] - 6), min(12 * h, hi[2] - lo[2] - 6)])
        p[: n // 50 + 1] += 1000.0                     # outside the grid
        p[n // 2] = p[n // 3]                          # two points in one place: not a pair
    return p.astype(np.float32)


@pytest.mark.parametrize("kind", ["thin", "dense", "clump", "column"])
@pytest.mark.parametrize("cell_h", [1.07, 1.9, 2.0, 15.0, 0.75, 0.4])   # cell edge in h: gridSrch 2, 2, 2, 2, 3, 6
@pytest.mark.parametrize("n", [1, 31, 33, 1500])
def test_density_and_pairs_equal_the_oracle(kind, cell_h, n):
    lo, hi = (-30.0, 0.0, -30.0), (30.0, 60.0, 30.0)
    p = scenes.make_params(lo, hi, grid_density=1.5 / cell_h)
    pos = cloud(kind, n, p.psmoothradius / p.sim_scale, lo, hi, seed=n)
    rng = np.random.default_rng(7)
    vel = rng.normal(0, 0.3, (n, 3)).astype(np.float32)
    clr = np.arange(n, dtype=np.uint32)
    with F.FluidSystem(p, n) as s:
        s.SetParticles(pos, vel, vel, clr=clr)
        s.InsertParticlesCUDA(); s.PrefixSumCellsCUDA(); s.CountingSortFullCUDA()
        s.ComputePressureCUDA(); s.ComputeForceCUDA()
        s.Sync()
        got = s.state()
    ref = O.State.new(p, pos, vel, vel, clr)
    O.insert(p, ref); O.prefix_sum(p, ref); O.counting_sort(p, ref); O.density(p, ref); O.force(p, ref)
    assert_bit_equal(got["clr"], ref.clr, f"{kind} {cell_h} {n}: order")
    assert_bit_equal(got["press"], ref.press, f"{kind} {cell_h} {n}: density")
    assert_bit_equal(got["force"], ref.force, f"{kind} {cell_h} {n}: force")
