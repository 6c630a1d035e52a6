"""Dirichlet conditions of small meshes, whose sweeps take them as an array over the field: it is filled for the next
step, not by each call that sets a condition, and it follows every change, alone, in a batch and between steps
and single solves.  Compared with the staged sweeps and their overwrites, bit by bit."""

import numpy as np
import pytest
import torch

from parabiofvm_b200 import Batch, Solver

pytestmark = pytest.mark.gpu


def _solver(grid, S, seed=0):
    rng = np.random.default_rng(seed)
    s = Solver(len(grid), (0,) * 3, tuple(20 * g for g in grid), (20,) * 3, rng.uniform(1e3, 1e5, S), [0.1] * S, 0.02)
    s.store_densities(rng.random(int(np.prod(grid)) * S, dtype=np.float32))
    return s


def _conditions(grid, S, seed):
    rng = np.random.default_rng(seed)
    inner = np.stack([rng.integers(0, g, 50) for g in grid], axis=1)
    faces = [(d, m, rng.random(S), rng.random(S) < 0.6) for d in range(len(grid)) for m in (False, True)]
    return faces, (inner, rng.random((50, S)), rng.random((50, S)) < 0.7)


def test_the_array_is_filled_once_for_the_next_step():
    grid, S = (40, 41, 42), 4
    s = _solver(grid, S)
    faces, inner = _conditions(grid, S, 1)
    counts = [s.launch_count]
    for _ in range(2):
        for f in faces:
            s.set_boundary_dirichlet(*f)
        s.set_interior_dirichlet(*inner)
        counts.append(s.launch_count)
        s.run_steps(1, 1)
        counts.append(s.launch_count)
        s.run_steps(1, 1)
        counts.append(s.launch_count)
    set1, first1, next1, set2, first2, next2 = np.diff(counts)
    assert set1 == set2 == 0 and next1 == next2
    assert first1 == first2 == next1 + 4  # the array, and the mask words of three axes
    s.close()


@pytest.mark.parametrize("grid,S", [((33, 20, 17), 4), ((40, 31), 3), ((600, 9, 8), 2)])
def test_changes_are_followed(grid, S):
    a, b = _solver(grid, S), _solver(grid, S)
    b.set_option("tma_prefetch", 1)
    if max(grid) > 512:  # lines that the staged sweep takes in chunks, which agree to rounding only
        b.set_option("tma_sweeps", 0)
    for s in (a, b):
        faces, inner = _conditions(grid, S, 1)
        for f in faces:
            s.set_boundary_dirichlet(*f)
        s.run_steps(2, 0)
        s.set_interior_dirichlet(*inner)
        s.diffusion()
        s.run_steps(1, 5)
        faces, inner = _conditions(grid, S, 2)
        s.set_boundary_dirichlet(*faces[1])
        s.set_interior_dirichlet(*inner)
        s.diffusion_gradient()
        s.set_boundary_dirichlet(0, False, None, None)
        s.run_steps(2, 9)
        s.set_interior_dirichlet(np.zeros((0, len(grid)), np.int32), np.zeros((0, S)), np.zeros((0, S)))
        for d in range(len(grid)):
            for m in (False, True):
                s.set_boundary_dirichlet(d, m, None, None)
        s.run_steps(1, 1)
        s.set_boundary_dirichlet(*faces[0])
        s.run_steps(1, 1)
    np.testing.assert_array_equal(a.load_densities(), b.load_densities())
    np.testing.assert_array_equal(a.load_gradients(), b.load_gradients())
    a.close()
    b.close()


def test_changes_are_followed_in_a_batch():
    """One member's lines are longer than the ensemble's kernels take: it steps by itself inside the batch."""
    shapes = [((600, 9, 8), 2), ((20, 21, 22), 3)]
    alone, members = ([_solver(g, S, seed=k) for k, (g, S) in enumerate(shapes)] for _ in range(2))
    batch = Batch(members)
    for seed in (1, 2):
        for group in (alone, members):
            for s, (g, S) in zip(group, shapes):
                faces, inner = _conditions(g, S, seed)
                for f in faces:
                    s.set_boundary_dirichlet(*f)
                s.set_interior_dirichlet(*inner)
        batch.run_steps(3, 0)
        for s in alone:
            s.run_steps(3, 0)
    batch.synchronize()
    for s, m in zip(alone, members):
        np.testing.assert_array_equal(s.load_densities(), m.load_densities())
        np.testing.assert_array_equal(s.load_gradients(), m.load_gradients())
    batch.close()
    for s in alone + members:
        s.close()


def test_a_caller_s_capture_before_any_step():
    """Inside a capture nothing is filled: the captured diffusion overwrites from the list."""
    grid, S = (33, 20, 17), 4
    a, b = _solver(grid, S), _solver(grid, S)
    stream = torch.cuda.Stream()
    for s in (a, b):
        faces, inner = _conditions(grid, S, 3)
        for f in faces:
            s.set_boundary_dirichlet(*f)
        s.set_interior_dirichlet(*inner)
    a.set_stream(stream.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        a.diffusion()
    for _ in range(3):
        graph.replay()
        b.diffusion()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(a.load_densities(), b.load_densities())
    a.close()
    b.close()
