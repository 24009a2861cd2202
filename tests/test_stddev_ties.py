"""Std-dev decisions at the threshold: the reference's sum over a whole cell of
up to 16^3 voxels is exact, builds whose cells tie with the threshold or lie
one unit beside it match the oracle, and ties cost such cells no loops."""
from __future__ import annotations

from fractions import Fraction

import numpy as np
import pytest


def _reference_sum(v):
    """Grid::stddev_scan's sequential double sum over (n, 4) voxels."""
    n = float(len(v))
    d = v.astype(np.float64) - v.sum(0).astype(np.float64) / n
    t = d * d
    return np.add.accumulate(((t[:, 0] + t[:, 1]) + t[:, 2]) + t[:, 3])[-1]


@pytest.mark.parametrize("side", [2, 4, 8, 16])
def test_the_sum_over_a_small_cell_is_exact(side):
    n = side ** 3
    rng = np.random.default_rng(side)
    cells = [np.where(rng.random((n, 4)) < f, hi, lo) for f in (0.5, 0.01, 0.37) for lo, hi in ((0, 255), (7, 8))]
    cells += [rng.integers(0, 256, (n, 4)) for _ in range(20)]
    cells.append(np.repeat(np.arange(n)[:, None] % 2 * 255, 4, 1))  # the largest sum there is
    for v in cells:
        E = int(n * (v.astype(object) ** 2).sum() - (v.sum(0).astype(object) ** 2).sum())
        assert Fraction(float(_reference_sum(v))) == Fraction(E, n)


def _tied(n, block, seed=3):
    """Blocks of voxels alternating by +-2 about a value of the block's own:
    every cell of 2 voxels a side up to the block's has deviation 2."""
    z, y, x = np.indices((n, n, n))
    k = -(-n // block)
    base = np.random.default_rng(seed).integers(1, 25, (k, k, k)) * 10 - 5
    g = np.zeros((n, n, n, 4), np.uint8)
    g[..., 0] = base[z // block, y // block, x // block] + 4 * ((x + y + z) & 1) - 2
    g[..., 3] = 255
    return g


@pytest.mark.gpu
@pytest.mark.parametrize("svo_type", ["sparse", "rope", "dag"])
@pytest.mark.parametrize("n,block", [(8, 8), (32, 4), (32, 16), (48, 16), (40, 8), (64, 32)])
def test_ties_match_the_oracle(ctx, svo_type, n, block):
    import oracle
    g = _tied(n, block)
    for threshold in (2.0, np.nextafter(2.0, 0), np.nextafter(2.0, 3)):
        ref, rstats = oracle.build_svo(g, svo_type, "std-dev", threshold)
        got, stats = ctx.build_svo(g, svo_type, "std-dev", threshold)
        assert stats == rstats
        assert np.array_equal(got, ref)


@pytest.mark.gpu
@pytest.mark.parametrize("side", [2, 4, 8, 16, 32])
def test_thresholds_of_a_cell_match_the_oracle(ctx, side):
    """The deviation of one cell of a random grid, and the doubles beside it."""
    import oracle
    rng = np.random.default_rng(side)
    g = rng.integers(90, 170, (32, 32, 40, 4)).astype(np.uint8)
    cell = g[:side, :side, :side].reshape(-1, 4)
    sd = np.sqrt(_reference_sum(cell) / float(len(cell)))
    for threshold in (sd, np.nextafter(sd, 0), np.nextafter(sd, 1e9)):
        for svo_type in ("sparse", "dag"):
            ref, rstats = oracle.build_svo(g, svo_type, "std-dev", float(threshold))
            got, stats = ctx.build_svo(g, svo_type, "std-dev", float(threshold))
            assert stats == rstats
            assert np.array_equal(got, ref)


@pytest.mark.gpu
def test_ties_of_small_cells_cost_no_loops(ctx):
    """256^3 voxels whose cells of 2 to 16 voxels a side all tie, against the
    same build with none (measured: 245 times as long with a loop per cell)."""
    import time
    import torch
    d = torch.from_numpy(_tied(256, 16)).cuda()
    torch.cuda.synchronize()

    def build(threshold):
        best = float("inf")
        for _ in range(4):
            t = time.perf_counter()
            ctx.build_svo_volume(d.data_ptr(), (256, 256, 256), "sparse", "std-dev", threshold, lean=True)[0].release()
            best = min(best, time.perf_counter() - t)
        return best

    assert build(2.0) <= 20 * build(3.0)
