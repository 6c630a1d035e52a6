"""Small meshes large enough that a CTA sweeps several tiles in turn (its tables staged once, carries and row
buffers used again), the last of them partly empty, on every axis and for lines of up to 32 blocks; and 3-D meshes
with an axis of one voxel, which take the other kernels.  The launches of a step tell which kernels ran: one a
sweep and the gradient in the small form, the overwrites besides in the other.  The same bits as the staged
sweeps, or for lines beyond 512 the direct ones."""

import numpy as np
import pytest

from gpu_runner import gpu_runner
from parabiofvm_b200 import Solver
from scenarios import make_oracle, rel_err
from test_gpu_parity import _box

pytestmark = pytest.mark.gpu


def _solver(grid, S, conditions):
    rng = np.random.default_rng(sum(grid) + S)
    dims = len(grid)
    s = Solver(dims, (0,) * 3, tuple(20 * g for g in grid), (20,) * 3, np.exp(rng.uniform(np.log(1e2), np.log(1e6), S)),
               rng.uniform(0.01, 1, S), 0.05)
    s.store_densities(rng.random(int(np.prod(grid)) * S, dtype=np.float32))
    if conditions:
        for d in range(dims):
            for m in (False, True):
                s.set_boundary_dirichlet(d, m, rng.random(S), rng.random(S) < 0.5)
        inner = np.stack([rng.integers(0, g, 500) for g in grid], axis=1)
        s.set_interior_dirichlet(inner, rng.random((500, S)), rng.random((500, S)) < 0.6)
    return s


def _launches(s):
    s.run_steps(1, 1)
    before = s.launch_count
    s.run_steps(1, 1)
    return s.launch_count - before


@pytest.mark.parametrize("grid,S", [((127, 126, 125), 4), ((215, 214, 213), 1), ((81, 79, 80), 8), ((139, 138, 137), 3),
                                    ((67, 65, 66), 16), ((45, 47, 46), 21), ((700, 120, 90), 1), ((90, 700, 120), 1),
                                    ((120, 90, 700), 1), ((1000, 1001), 4)])
@pytest.mark.parametrize("conditions", [False, True])
def test_several_tiles_a_cta(grid, S, conditions):
    a, b = _solver(grid, S, conditions), _solver(grid, S, conditions)
    b.set_option("tma_prefetch", 1)
    if max(grid) > 512:
        b.set_option("tma_sweeps", 0)
    assert _launches(a) == len(grid) + 1  # within the small form's limits, whatever these become
    if conditions:
        assert _launches(b) > len(grid) + 1
    else:
        b.run_steps(2, 1)
    np.testing.assert_array_equal(a.load_densities(), b.load_densities())
    np.testing.assert_array_equal(a.load_gradients(), b.load_gradients())
    a.close()
    b.close()


@pytest.mark.parametrize("grid", [(1, 30, 40), (40, 1, 30), (30, 40, 1), (1, 1, 50), (50, 1, 1)])
def test_axis_of_one_voxel(grid):
    w = _box((5, 5, 5), 4, seed=1)
    w.bbox_max = tuple(20 * g for g in grid)
    w.densities = np.random.default_rng(2).random(int(np.prod(grid)) * 4).astype(np.float32)
    w.interior_voxels = w.interior_values = w.interior_conditions = None
    o, g = make_oracle(w, np.float32), gpu_runner(w)
    o.run_steps(3, 0)
    g.run_steps(3, 0)
    assert _launches(g.s) > 4
    o.run_steps(2, 1)
    assert rel_err(g.densities(), o.densities()) < 1e-5
    g.close()
