"""Binnings that follow one another in the same scratch: each must find it as the one before was meant to leave it.
Agents that move between them, at the sizes where the binning changes form and tiles, counts that shrink within the
storage past those sizes, and key spaces of one digit of the radix passes to three.  Checked through the
update against the voxel sums in numpy, with rates whose sums are exact in float32 (the field then matches to the
rounding of the update's three operations, 4e-7)."""

import numpy as np
import pytest

from parabiofvm_b200 import Solver

pytestmark = pytest.mark.gpu

S, DX = 2, 16  # voxel volume 4096 and agents of volume 4096: the terms are the rates themselves
BLOCK, SMALL_TILES = 16384, 1 << 18


def _check(s, grid, rng, sec, upt, pos):
    V = int(np.prod(grid))
    field = rng.integers(0, 64, (V, S)).astype(np.float32) / 8
    s.store_densities(field)
    s.secretion(True)
    got = s.load_densities().reshape(V, S)
    cell = (pos / np.float32(DX)).astype(np.int64)
    v = cell[:, 0] + grid[0] * (cell[:, 1] + grid[1] * cell[:, 2])
    num, den, hit = np.zeros((V, S)), np.ones((V, S)), np.zeros(V, bool)
    np.add.at(num, v, sec)
    np.add.at(den, v, sec + upt)
    hit[v] = True
    want = np.where(hit[:, None], (field + num) / den, field)
    np.testing.assert_array_equal(got[~hit], field[~hit])
    assert np.abs(got - want).max() <= 4e-7 * max(1.0, np.abs(want).max())


def _agents(rng, grid, n):
    pos = (rng.random((n, 3)) * np.array(grid) * DX).astype(np.float32)
    pos = np.minimum(pos, np.nextafter(np.array(grid, np.float32) * DX, np.float32(0)))
    sec, upt = (rng.integers(0, 4, (n, S)).astype(np.float32) / 16 for _ in range(2))
    return sec, upt, pos


def _store(s, sec, upt, pos):
    one, zero = np.ones_like(sec), np.zeros_like(sec)
    s.store_agents(sec, one, upt, zero, zero, None, np.full(len(pos), float(DX ** 3), np.float32), pos)


# 1 to 1,023 voxels: one digit; 1,024 to 2^20 - 1: two; from 2^20: three
@pytest.mark.parametrize("grid", [(9, 8, 7), (40, 30, 20), (128, 96, 90), (101, 102, 103)])
@pytest.mark.parametrize("internalized", [False, True])
def test_binnings_in_the_same_scratch(grid, internalized):
    rng = np.random.default_rng(sum(grid))
    s = Solver(3, (0, 0, 0), tuple(g * DX for g in grid), (DX,) * 3, [1.0] * S, [0.0] * S, 1.0,
               compute_internalized=internalized)
    for n in (SMALL_TILES + 1, SMALL_TILES, SMALL_TILES - 1023, 200_000, BLOCK + 1, BLOCK, 1025, BLOCK + 1, SMALL_TILES + 1):
        sec, upt, pos = _agents(rng, grid, n)
        _store(s, sec, upt, pos)
        _check(s, grid, rng, sec, upt, pos)
        for _ in range(2):
            pos = _agents(rng, grid, n)[2]
            s.store_agent_positions(pos)
            _check(s, grid, rng, sec, upt, pos)
    s.close()
