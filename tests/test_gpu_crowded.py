"""Agents crowded into few voxels, binned by one CTA: segments around the length from which their terms are spread
over a CTA's threads, several such segments in one CTA and across CTAs, beside short ones, one and four substrates
a thread, agents outside the mesh.  Fields and amounts are the oracle's bits, and binning again costs no more
than the update itself takes."""

import numpy as np
import pytest
import torch

from scenarios import make_gpu, make_oracle
from parabiofvm_b200 import Solver
from parabiofvm_b200.workloads import Agents, Scenario

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [1, 3, 4, 8, 33])
@pytest.mark.parametrize("lengths", [[32], [33], [31, 32, 33, 34], [1] * 40 + [33] * 70 + [2] * 30 + [257, 256, 255] + [1] * 9,
                                     [2000, 1, 40, 1500, 1, 1], [40] * 300])
def test_crowded_voxels_against_the_oracle(S, lengths):
    rng = np.random.default_rng(S + len(lengths))
    g = (9, 8, 7)
    n = int(sum(lengths))
    voxel = np.repeat(rng.permutation(int(np.prod(g)))[:len(lengths)], lengths)
    at = np.stack([voxel % g[0], voxel // g[0] % g[1], voxel // (g[0] * g[1])], axis=1)
    pos = (at + rng.uniform(0.1, 0.9, (n, 3))) * 20
    pos = pos[rng.permutation(n)]
    w = Scenario(dims=3, bbox_min=(0, 0, 0), bbox_max=tuple(20 * v for v in g), voxel_shape=(20, 20, 20),
                 diffusion_coefficients=[1e4] * S, decay_rates=[0.1] * S, time_step=0.01, initial_conditions=[1.0] * S)
    w.compute_internalized = True
    r = lambda *s: rng.random(s).astype(np.float32)  # noqa: E731
    w.densities = r(int(np.prod(g)) * S)
    w.agents = Agents(secretion_rates=r(n, S), saturation_densities=r(n, S), uptake_rates=r(n, S),
                      net_export_rates=r(n, S), internalized=r(n, S), fraction_released=r(n, S),
                      volumes=np.full(n, 1000.0), positions=pos)
    o, s = make_oracle(w, np.float32), make_gpu(w)
    for recompute in (True, False):
        o.secretion(recompute)
        s.secretion(recompute)
    np.testing.assert_array_equal(s.load_densities(), np.asarray(o.densities(), np.float32).reshape(-1))
    np.testing.assert_array_equal(s.load_internalized(), np.asarray(o.internalized(), np.float32).reshape(-1))
    s.close()


def test_binning_a_crowd_costs_no_more_than_its_update():
    """16,384 agents in one voxel: the update walks them one after another; binning them again may take as long
    once more, not several times."""
    A, S = 16_384, 4
    rng = np.random.default_rng(0)
    s = Solver(3, (0,) * 3, (600,) * 3, (20,) * 3, [1e4] * S, [0.1] * S, 0.01, compute_internalized=True)
    stream = torch.cuda.Stream()
    s.set_stream(stream.cuda_stream)
    zero = np.zeros((A, S), np.float32)
    s.store_agents(*[rng.random((A, S), dtype=np.float32) for _ in range(3)], zero, zero, None,
                   np.full(A, 1000.0, np.float32), np.full((A, 3), 310.0, np.float32))

    def timed(recompute):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        for k in range(6):
            if k == 1:
                a.record(stream)
            s.secretion(recompute)
        b.record(stream)
        b.synchronize()
        return a.elapsed_time(b) / 5

    rebinning, update = timed(True), timed(False)
    assert rebinning < 2 * update, (rebinning, update)
    s.close()
