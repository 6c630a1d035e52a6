"""The gradient kernel's column arithmetic (a multiplication in place of the divisions by row and substrates) and
its marches: rows and substrate counts that are powers of two, one less and one more, axes of one and two voxels,
last marches of few planes, 1-D to 3-D.  The same bits as the formula in numpy.  And a 2-D gradient moves its
bytes at a fair share of a device copy's rate."""

import numpy as np
import pytest
import torch

from parabiofvm_b200 import Solver

pytestmark = pytest.mark.gpu

SHAPES = [((1,), 1), ((2,), 3), ((2047,), 5), ((2048,), 1), ((1, 1), 2), ((1, 9), 1), ((255, 3), 1), ((256, 257), 1),
          ((257, 255), 1), ((1023, 5), 3), ((64, 33), 4), ((2000, 31), 7), ((1, 1, 1), 4), ((5, 1, 3), 1), ((3, 5, 1), 8),
          ((2, 2, 2), 4), ((33, 31, 3), 4), ((31, 33, 5), 3), ((500, 500, 9), 4), ((300, 401, 10), 4), ((129, 65, 17), 16),
          ((7, 6, 1999), 1), ((4, 3, 2000), 4)]


def _solver(grid, S):
    s = Solver(len(grid), (0,) * 3, tuple(20 * g for g in grid), (20,) * 3, [1e4] * S, [0.1] * S, 0.01)
    field = np.random.default_rng(sum(grid) + S).random(int(np.prod(grid)) * S, dtype=np.float32)
    s.store_densities(field)
    return s, field.reshape(tuple(reversed(grid)) + (S,))


@pytest.mark.parametrize("grid,S", SHAPES)
def test_gradient_bits(grid, S):
    s, u = _solver(grid, S)
    s.gradient()
    want = []
    for d, n in enumerate(grid):
        w = np.moveaxis(u, len(grid) - 1 - d, 0)
        g = np.zeros_like(u)
        t = np.moveaxis(g, len(grid) - 1 - d, 0)
        if n > 1:
            t[1:-1] = (w[2:] - w[:-2]) * np.float32(1 / 40)
            t[0] = (w[1] - w[0]) * np.float32(1 / 20)
            t[-1] = (w[-1] - w[-2]) * np.float32(1 / 20)
        want.append(g)
    want = np.stack(want, axis=0 if len(grid) == 3 else -1)
    np.testing.assert_array_equal(s.load_gradients(), want.reshape(-1))
    s.close()


def test_gradient_of_a_large_slice_keeps_its_rate():
    """2000 x 2000 x 4: 192 MB read and written; a device copy that moves as much is the measure."""
    s, _ = _solver((2000, 2000), 4)
    stream = torch.cuda.Stream()
    s.set_stream(stream.cuda_stream)
    a = torch.zeros(24_000_000, device="cuda")
    b = torch.empty_like(a)
    torch.cuda.synchronize()

    def best(f):
        times = []
        with torch.cuda.stream(stream):
            for _ in range(5):
                e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                f()
                e0.record()
                for _ in range(20):
                    f()
                e1.record()
                e1.synchronize()
                times.append(e0.elapsed_time(e1) / 20)
        return min(times)

    copy, gradient = best(lambda: b.copy_(a)), best(s.gradient)
    assert gradient < 2.05 * copy, (gradient, copy)
    s.close()
