"""Solvers in threads of their own whose sweeps are the same kernel with different amounts of shared memory:
one thread's launch must not change what the other's may use.  Results are those of one thread alone."""

import threading

import numpy as np
import pytest

from parabiofvm_b200 import Solver

pytestmark = pytest.mark.gpu


def _solver(grid, S, staged):
    s = Solver(3, (0,) * 3, tuple(g * 20 for g in grid), (20,) * 3, [1e4] * S, [0.1] * S, 0.01)
    if staged:
        s.set_option("tma_prefetch", 1)  # the staged sweeps also where the mesh is small
    s.store_densities(np.random.default_rng(grid[0]).random(int(np.prod(grid)) * S, dtype=np.float32))
    return s


@pytest.mark.parametrize("grids,S,staged", [(((512, 5, 4), (380, 5, 4)), 1, False), (((512, 8, 8), (256, 8, 8)), 4, True)])
def test_two_threads_with_solvers_of_their_own(grids, S, staged):
    calls = 3000
    want = []
    for g in grids:
        s = _solver(g, S, staged)
        for _ in range(calls):
            s.diffusion()
        want.append(s.load_densities())
        s.close()
    solvers = [_solver(g, S, staged) for g in grids]
    errors, start = [], threading.Barrier(2)

    def work(s):
        start.wait()
        try:
            for _ in range(calls):
                s.diffusion()
        except Exception as e:  # noqa: BLE001 (reported by the assertion below)
            errors.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in solvers]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for s, w in zip(solvers, want):
        np.testing.assert_array_equal(s.load_densities(), w)
        s.close()
