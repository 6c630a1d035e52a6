"""The binning at the sizes where it changes form: one CTA up to 16,384 agents, look-back tiles of 1,024
keys up to 2^18 agents and of 4,096 beyond, a key space of one, two and three radix digits, agents
outside the mesh.  Checked through one secretion step against the voxel sums in numpy: with uptake and
secretion of exact binary fractions every sum is exact in float32, whatever the order, so the field
must match to the rounding of the update itself (three operations, 4e-7)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("agents", [1, 1023, 1025, 16384, 16385, 17408, (1 << 18), (1 << 18) + 1])
@pytest.mark.parametrize("grid", [(5, 4, 3), (40, 30, 20), (70, 64, 65)])
def test_voxel_sums_at_the_edges_of_the_forms(agents, grid):
    from parabiofvm_b200 import Solver
    from parabiofvm_b200._abi import BfvmError

    rng = np.random.default_rng(agents + grid[0])
    S, dx = 2, 16  # voxel volume 4096, volumes 4096: the terms are the rates themselves
    s = Solver(3, (0, 0, 0), tuple(g * dx for g in grid), (dx,) * 3, [1.0, 1.0], [0.0, 0.0], 1.0)
    V = int(np.prod(grid))
    field = rng.integers(0, 64, (V, S)).astype(np.float32) / 8
    s.store_densities(field)
    pos = (rng.random((agents, 3)) * np.array(grid) * dx).astype(np.float32)
    pos = np.minimum(pos, np.nextafter(np.array(grid, np.float32) * dx, np.float32(0)))
    outside = rng.random(agents) < 0.01
    pos[outside] = -2.0 * dx
    sec = rng.integers(0, 4, (agents, S)).astype(np.float32) / 16
    upt = rng.integers(0, 4, (agents, S)).astype(np.float32) / 16
    sat = np.ones((agents, S), np.float32)
    zero = np.zeros((agents, S), np.float32)
    s.store_agents(sec, sat, upt, zero, zero, None, np.full(agents, float(dx ** 3), np.float32), pos)
    s.secretion(True)
    if outside.any():
        with pytest.raises(BfvmError):
            s.synchronize()
    got = s.load_densities().reshape(V, S)
    cell = (pos[~outside] / np.float32(dx)).astype(np.int64)
    v = cell[:, 0] + grid[0] * (cell[:, 1] + grid[1] * cell[:, 2])
    num, den = np.zeros((V, S)), np.ones((V, S))
    np.add.at(num, v, sec[~outside])
    np.add.at(den, v, (sec + upt)[~outside])
    hit = np.zeros(V, bool)
    hit[v] = True
    want = np.where(hit[:, None], (field + num) / den, field)
    assert np.array_equal(got[~hit], field[~hit])
    assert np.abs(got - want).max() <= 4e-7 * max(1.0, np.abs(want).max())
    s.close()
