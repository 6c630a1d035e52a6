"""Which staged sweeps pair their tiles by default: never a choice that is slower than both options, on lines of few
blocks in fields of few tiles, where the z sweep lost its pairing once.  Times of the same sweep in one process."""

import numpy as np
import pytest
import torch

from parabiofvm_b200 import BfvmError, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,S,axis", [((70, 70, 128), 8, 2), ((80, 64, 128), 8, 2), ((200, 200, 350), 4, 2),
                                         ((80, 128, 64), 8, 1), ((300, 300, 300), 4, 1), ((320, 320, 320), 4, 2)])
def test_default_pairing_is_the_faster_one(grid, S, axis):
    s = Solver(3, (0,) * 3, tuple(20 * g for g in grid), (20,) * 3, [1e4] * S, [0.1] * S, 0.01)
    stream = torch.cuda.Stream()
    s.set_stream(stream.cuda_stream)
    s.store_densities(np.random.default_rng(1).random(int(np.prod(grid)) * S, dtype=np.float32))

    def best():
        times = []
        for _ in range(6):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            s.sweep(axis)
            e0.record(stream)
            for _ in range(30):
                s.sweep(axis)
            e1.record(stream)
            e1.synchronize()
            times.append(e0.elapsed_time(e1) / 30)
        return min(times)

    default = best()
    options = []
    for pairs in (0, 2):
        s.set_option("tma_pairs", pairs)
        options.append(best())
    assert default <= 1.08 * min(options), (default, options)  # 12 % where it was lost; runs differ by 2 %
    s.close()


def test_default_can_be_put_back():
    w = np.random.default_rng(2).random(40 * 70 * 128 * 8, dtype=np.float32)
    fields = []
    for values in ((), (2, -1), (0,)):
        s = Solver(3, (0,) * 3, (800, 1400, 2560), (20,) * 3, [1e4] * 8, [0.1] * 8, 0.01)
        for v in values:
            s.set_option("tma_pairs", v)
        for v in (-2, 3):
            with pytest.raises(BfvmError):
                s.set_option("tma_pairs", v)
        s.store_densities(w)
        s.sweep(2)
        fields.append(s.load_densities())
        s.close()
    for f in fields[1:]:
        np.testing.assert_array_equal(f, fields[0])
