"""The ensemble sweeps' two forms of the solve (a mesh alone whose rows the copy engine does not take, and batches):
the same bits, for lines of one to sixteen blocks and substrate counts that leave lanes idle or fill them.  And on
one mesh the x sweep, which once spilled and staged slowly, keeps its time beside the z sweep's."""

import numpy as np
import pytest
import torch

from parabiofvm_b200 import Batch, Solver

pytestmark = pytest.mark.gpu


def _solver(grid, S):
    rng = np.random.default_rng(sum(grid) + S)
    s = Solver(3, (0,) * 3, tuple(20 * g for g in grid), (20,) * 3, np.exp(rng.uniform(np.log(1e2), np.log(1e6), S)),
               rng.uniform(0.01, 1, S), 0.05)
    s.store_densities(rng.random(int(np.prod(grid)) * S, dtype=np.float32))
    return s


@pytest.mark.parametrize("grid,S", [((5, 44, 40), 5), ((31, 65, 33), 1), ((49, 50, 51), 17), ((97, 33, 12), 7),
                                    ((501, 9, 10), 3), ((10, 511, 7), 9), ((9, 11, 480), 32), ((63, 129, 257), 2)])
def test_alone_and_in_a_batch(grid, S):
    alone, members = [_solver(grid, S), _solver((6, 7, 8), 3)], [_solver(grid, S), _solver((6, 7, 8), 3)]
    alone[0].set_option("tma_sweeps", 0)
    b = Batch(members)
    b.run_steps(2, 1)
    b.synchronize()
    for s, m in zip(alone, members):
        s.run_steps(2, 1)
        np.testing.assert_array_equal(s.load_densities(), m.load_densities())
        np.testing.assert_array_equal(s.load_gradients(), m.load_gradients())
    b.close()
    for s in alone + members:
        s.close()


def test_x_sweep_of_one_mesh_keeps_its_time():
    s = _solver((101, 103, 97), 9)
    stream = torch.cuda.Stream()
    s.set_stream(stream.cuda_stream)

    def best(axis):
        times = []
        for _ in range(6):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            s.sweep(axis)
            e0.record(stream)
            for _ in range(40):
                s.sweep(axis)
            e1.record(stream)
            e1.synchronize()
            times.append(e0.elapsed_time(e1) / 40)
        return min(times)

    x, z = best(0), best(2)
    assert x < 1.16 * z, (x, z)  # 1.21 with that form, 1.07 to 1.09 without
    s.close()
