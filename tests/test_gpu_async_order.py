"""The order that the asynchronous agent copies promise a caller with a stream of its own: run_steps waits for
them on the GPU, so once that stream is through, the host buffer holds the copy, also when no step rebinned.
32 MB to the host take several times as long as the step."""

import numpy as np
import pytest
import torch

from parabiofvm_b200 import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [1, 3])
def test_run_steps_without_rebinning_waits_for_copies(steps):
    edge, S, A = 64, 8, 1_000_000
    rng = np.random.default_rng(steps)
    s = Solver(3, (0,) * 3, (edge * 20,) * 3, (20,) * 3, [1e4] * S, [0.1] * S, 0.01, compute_internalized=True)
    stream = torch.cuda.Stream()
    s.set_stream(stream.cuda_stream)
    s.store_densities(rng.random(edge ** 3 * S, dtype=np.float32))
    rates = [rng.random((A, S), dtype=np.float32) for _ in range(3)]
    amounts = rng.random((A, S), dtype=np.float32)
    pos = rng.random((A, 3), dtype=np.float32) * np.float32(edge * 20 - 1)
    s.store_agents(*rates, np.zeros((A, S), np.float32), amounts, None, np.full(A, 1000.0, np.float32), pos)
    s.run_steps(2, 0)  # both step graphs exist
    want = s.load_internalized().copy()
    got = torch.full((A * S,), -1.0, dtype=torch.float32, pin_memory=True).numpy()
    s.load_internalized_async(got)
    s.run_steps(steps, 1)
    stream.synchronize()
    last = got[-1024:].copy()  # at once: a copy of the whole on the host would give the transfer time to finish
    s.synchronize()
    assert np.array_equal(last, want[-1024:])
    assert np.array_equal(got, want)
    s.close()
