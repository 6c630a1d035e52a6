"""The staged sweeps' launch shapes on meshes that the small form leaves to them: tuned shapes, chunks of long lines
(asked for, or in fields beyond the small form), lines of 5 and 6 blocks with four groups a CTA and paired tiles,
faces by position and the slab solve at more than 640 threads.  The launches of a step tell which path ran."""

import numpy as np
import pytest

from gpu_runner import gpu_runner
from parabiofvm_b200 import Solver
from scenarios import make_oracle, rel_err
from test_gpu_parity import _box
from test_gpu_slabs import _run, _single, _workload

pytestmark = pytest.mark.gpu

STAGED = 8  # launches of a 3-D step with conditions: four overwrites, three sweeps, the gradient


def _launches(s):
    s.run_steps(1, 1)
    before = s.launch_count
    s.run_steps(1, 1)
    return s.launch_count - before


def _plain(grid, S):
    rng = np.random.default_rng(sum(grid) + 7 * S)
    s = Solver(3, (0,) * 3, tuple(20 * g for g in grid), (20,) * 3, np.exp(rng.uniform(np.log(1e2), np.log(1e6), S)),
               rng.uniform(0.01, 1, S), 0.05)
    s.store_densities(rng.random(int(np.prod(grid)) * S, dtype=np.float32))
    return s


@pytest.mark.parametrize("edge,S", [(96, 8), (152, 3)])
def test_tuned_shapes_keep_results(edge, S):
    w = _box((edge, edge, edge), S, seed=edge + S)
    ref, tuned = gpu_runner(w), gpu_runner(w)
    assert _launches(ref.s) == STAGED
    choices = tuned.s.autotune()
    assert all(1 <= groups <= 8 and 2 <= stages <= 4 for groups, stages in choices)
    assert _launches(tuned.s) == STAGED
    later = gpu_runner(w)  # of the same shape: takes the cached choice
    later.run_steps(2, 1)
    for r in (tuned, later):
        np.testing.assert_array_equal(r.densities(), ref.densities())
        np.testing.assert_array_equal(r.gradients(), ref.gradients())
    for r in (ref, tuned, later):
        r.close()


@pytest.mark.parametrize("grid,S", [((1024, 16, 16), 4), ((777, 12, 10), 4), ((700, 600, 4), 4), ((1000, 9, 30), 6)])
def test_chunks_asked_for(grid, S):
    """Against whole lines and the oracle to rounding, and their own bits again."""
    w = _box(grid, S, seed=7 * sum(grid) + S)
    cut, again, whole = gpu_runner(w), gpu_runner(w), gpu_runner(w)
    for r in (cut, again):
        r.s.set_option("chunk_elements", 512)
    whole.s.set_option("tma_sweeps", 0)
    o = make_oracle(w, np.float32)
    o.run_steps(2, 1)
    assert _launches(cut.s) > STAGED  # the chunks' sums and their combination
    again.run_steps(2, 1)
    whole.run_steps(2, 1)
    np.testing.assert_array_equal(cut.densities(), again.densities())
    assert rel_err(cut.densities(), whole.densities()) < 1e-5
    assert rel_err(cut.densities(), o.densities()) < 1e-5
    for r in (cut, again, whole):
        r.close()


# y and z lines are cut from 2^17 of them on
@pytest.mark.parametrize("grid,S,chunk", [((640, 160, 128), 4, 0), ((256, 640, 130), 4, 0), ((256, 130, 640), 4, 0),
                                          ((500, 96, 72), 4, 250), ((256, 300, 130), 4, 160), ((640, 160, 90), 8, 0)])
def test_chunks_of_large_fields(grid, S, chunk):
    """Each element goes through at most 640 multiply-adds of a line that damps its errors: 2e-5 of the largest
    value for the one step."""
    out, launches = [], []
    for staged in (1, 0):
        s = _plain(grid, S)
        s.set_option("chunk_elements", chunk if staged else 0)
        s.set_option("tma_sweeps", staged)
        s.diffusion()
        out.append(s.load_densities())
        launches.append(_launches(s))
        s.close()
    assert launches[0] > launches[1] == 4, launches
    assert np.abs(out[0] - out[1]).max() <= 2e-5 * np.abs(out[1]).max()


@pytest.mark.parametrize("grid,S", [((192, 180, 161), 4), ((130, 192, 190), 4), ((150, 129, 192), 3), ((96, 161, 192), 8)])
def test_lines_of_five_and_six_blocks(grid, S):
    out = []
    for option, value in (("tma_sweeps", 0), ("tma_pairs", -1), ("tma_pairs", 0), ("tma_pairs", 2)):
        s = _plain(grid, S)
        s.set_option(option, value)
        s.diffusion()
        out.append(s.load_densities())
        s.close()
    for o in out[1:]:
        np.testing.assert_array_equal(o, out[0])


@pytest.mark.parametrize("grid,S", [((250, 140, 131), 4), ((132, 224, 130), 4), ((130, 110, 250), 4), ((249, 80, 64), 8)])
def test_faces_by_position_at_seven_and_eight_blocks(grid, S):
    w = _box(grid, S, seed=sum(grid))
    for f, (vals, conds) in enumerate(w.boundary.values()):
        vals[:] = 10.0 * (f + 1) + np.arange(S)
        conds[:] = (np.arange(S) + f) % 3 > 0
    w.interior_voxels = w.interior_values = w.interior_conditions = None  # none may lie on a face
    runs = [gpu_runner(w) for _ in range(3)]
    runs[0].s.set_option("face_dirichlet", 1)
    runs[2].s.set_option("tma_sweeps", 0)
    assert _launches(runs[0].s) < _launches(runs[1].s)  # nothing is left to overwrite after the sweeps
    runs[2].run_steps(2, 1)
    for r in runs[1:]:
        np.testing.assert_array_equal(runs[0].densities(), r.densities())
    for r in runs:
        r.close()


def test_slabs_of_seven_and_eight_blocks():
    """120 x 120 x 4 lines: enough tiles for three groups a CTA; tolerances of the other slab tests."""
    w = _workload(120, 480, 4, 400, seed=11)
    dens, grad, _ = _run(w, [0, 224, 480], 2)
    ref = _single(w, 2)
    assert rel_err(dens, ref[0]) < 2e-5
    du = float(np.abs(dens.astype(np.float64) - ref[0]).max())
    dg = float(np.abs(grad.astype(np.float64) - ref[1]).max())
    assert dg <= 2 * du / w.voxel_shape[2] + 1e-6 * float(np.abs(ref[1]).max())
