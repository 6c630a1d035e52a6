"""Staged sweeps at launch shapes of more than 640 threads (lines of 7, 8 and 12 blocks of 32 in fields of
enough tiles) and at each substrate count whose x sweep transposes its stores: the same bits as the direct
kernels.  Chunks of long lines agree with whole lines to rounding: each element goes through at most 512
multiply-adds of a line that damps its errors, so 2e-5 of the largest value is ample."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,S,chunked", [((250, 140, 131), 4, False), ((224, 200, 221), 2, False),
                                            ((128, 384, 97), 4, False), ((132, 105, 384), 4, False),
                                            ((249, 80, 110), 8, False), ((219, 91, 80), 16, False),
                                            ((140, 250, 130), 4, False), ((141, 132, 199), 4, False),
                                            ((500, 96, 72), 4, True)])
def test_staged_shapes_same_bits_as_direct(grid, S, chunked):
    from parabiofvm_b200 import Solver

    rng = np.random.default_rng(sum(grid) + 7 * S)
    field = rng.random((int(np.prod(grid)), S)).astype(np.float32)
    D = np.exp(rng.uniform(np.log(1e2), np.log(1e6), S))
    lam = rng.uniform(0.01, 1, S)
    out = []
    for staged in (1, 0):
        s = Solver(3, (0,) * 3, tuple(g * 20 for g in grid), (20,) * 3, D, lam, 0.05)
        s.set_option("tma_sweeps", staged)
        s.store_densities(field)
        s.diffusion()
        out.append(s.load_densities())
        s.close()
    if chunked:
        assert np.abs(out[0] - out[1]).max() <= 2e-5 * np.abs(out[1]).max()
    else:
        assert np.array_equal(*out)
