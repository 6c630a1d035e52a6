"""The small-mesh kernels against the staged sweeps, the scattered overwrites and the plain gradient and
secretion launches (any option that names those selects them; results are the same bits): line lengths at
the edges of a block of 32, one to 32 blocks, every substrate count that has an instance of its own
and others, tiles with rows or columns missing, 1-D to 3-D, face and interior conditions that meet, and
agents; two steps, so that one of them rebins beside the diffusion."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [((2, 2, 2), 1), ((31, 5, 3), 2), ((32, 33, 2), 3), ((33, 32, 31), 4), ((64, 65, 3), 5), ((3, 64, 65), 6),
          ((97, 9, 34), 7), ((40, 41, 42), 8), ((65, 4, 40), 12), ((34, 33, 20), 16), ((36, 10, 7), 17),
          ((33, 6, 5), 32), ((512, 5, 4), 1), ((4, 512, 3), 4), ((3, 4, 500), 3), ((300, 257), 3), ((20, 700), 2),
          ((45, 31), 16), ((33, 5, 34), 9), ((21, 40, 9), 11), ((500,), 4), ((2,), 32), ((128, 100, 80), 8),
          ((513, 4, 3), 3), ((3, 700, 5), 4), ((4, 3, 1024), 2), ((1000, 30), 5), ((30, 999), 1), ((1024,), 6)]


@pytest.mark.parametrize("grid,S", SHAPES)
@pytest.mark.parametrize("conditions", ["none", "faces", "both"])
def test_small_mesh_same_bits_as_staged(grid, S, conditions):
    from parabiofvm_b200 import Solver

    dims, dx = len(grid), 20
    rng = np.random.default_rng(sum(grid) + 7 * S)
    V = int(np.prod(grid))
    field = rng.random((V, S)).astype(np.float32)
    D = np.exp(rng.uniform(np.log(1e2), np.log(1e6), S))
    lam = rng.uniform(0.01, 1, S)
    A = max(1, V // 10)
    pos = (rng.random((A, dims)) * np.array(grid) * dx * 0.999).astype(np.float32)
    rates = [rng.random((A, S)).astype(np.float32) for _ in range(3)]
    zero = np.zeros((A, S), np.float32)
    inner = np.stack([rng.integers(0, g, max(1, V // 50)) for g in grid], axis=1).astype(np.int32)
    ivals, iconds = rng.random((len(inner), S)), rng.random((len(inner), S)) < 0.6
    faces = [(d, m, rng.random(S), rng.random(S) < 0.5) for d in range(dims) for m in (False, True)]
    out = []
    for staged in (False, True):
        s = Solver(dims, (0,) * 3, tuple(g * dx for g in grid), (dx,) * 3, D, lam, 0.05, compute_internalized=True)
        if staged:
            s.set_option("tma_prefetch", 1)
            if max(grid) > 512:  # lines that the staged sweep takes in chunks, which agree to rounding only
                s.set_option("tma_sweeps", 0)
        if conditions != "none":
            for d, m, v, c in faces:
                s.set_boundary_dirichlet(d, m, v, c)
        if conditions == "both":
            s.set_interior_dirichlet(inner, ivals, iconds)
        s.store_densities(field)
        s.store_agents(*rates, zero, zero, None, np.full(A, 1000.0, np.float32), pos)
        s.run_steps(2, 0)
        out.append((s.load_densities(), s.load_gradients(), s.load_internalized()))
        s.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_condition_that_looks_like_none():
    """A Dirichlet value with the bits that mark "no condition" leaves the mesh to the overwrite kernels."""
    from parabiofvm_b200 import Solver

    mark = np.array([0xFFFFFFFF], np.uint32).view(np.float32)
    s = Solver(3, (0, 0, 0), (100, 100, 100), (20, 20, 20), [1000.0], [0.1], 0.01)
    s.set_interior_dirichlet(np.array([[2, 2, 2]], np.int32), mark, np.ones(1, np.uint8))
    s.store_densities(np.ones(125, np.float32))
    s.dirichlet()
    s.diffusion()
    assert np.isnan(s.load_densities()[62])
    s.close()
