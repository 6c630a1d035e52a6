"""The bounded waits of the agent binning, run out on purpose: the test-only options name a tile that never
publishes its count, so the tiles after it give up after the (short) limit and the kernels return.  The next
synchronising call reports BFVM_ERR_TIMEOUT once; field and internalized amounts are what the step without
secretion left (also through a release, an addition and a load before the report), and the solver then steps bit
for bit like one that was given that state."""

import numpy as np
import pytest

from parabiofvm_b200 import Batch, Solver
from parabiofvm_b200._abi import BfvmError

pytestmark = pytest.mark.gpu

BFVM_ERR_TIMEOUT = 7
A, S, EDGE = 40_000, 4, 40  # 40 tiles of 1,024 keys


def _state(seed):
    rng = np.random.default_rng(seed)
    return {"field": rng.random((EDGE ** 3, S), dtype=np.float32),
            "rates": [rng.random((A, S), dtype=np.float32) for _ in range(3)],
            "amounts": rng.random((A, S), dtype=np.float32), "released": rng.random((A, S), dtype=np.float32),
            "pos": rng.random((A, 3), dtype=np.float32) * np.float32(EDGE * 20 - 1)}


def _solver(d, internalized, field=None, amounts=None):
    s = Solver(3, (0,) * 3, (EDGE * 20,) * 3, (20,) * 3, [1e4] * S, [0.1] * S, 0.01, compute_internalized=internalized)
    s.store_densities(d["field"] if field is None else field)
    s.store_agents(*d["rates"], np.zeros((A, S), np.float32), d["amounts"] if amounts is None else amounts,
                   d["released"], np.full(A, 1000.0, np.float32), d["pos"])
    return s


def _same(a, b):
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


def _all(s):
    return s.load_densities(), s.load_gradients(), s.load_internalized()


@pytest.mark.parametrize("option", ["test_drop_bin_tile", "test_drop_segment_tile"])
@pytest.mark.parametrize("tile", [0, 17])
@pytest.mark.parametrize("internalized,binned_before", [(True, False), (True, True), (False, True)])
def test_binning_wait_runs_out_and_solver_recovers(option, tile, internalized, binned_before):
    d = _state(tile)
    s = _solver(d, internalized)
    if binned_before:
        s.run_steps(3, 0)
    field, _, amounts = _all(s)
    s.set_option("wait_limit_cycles", 2_000_000)  # about a millisecond
    s.set_option(option, tile)
    with pytest.raises(BfvmError) as e:
        s.run_steps(2, 0)
        s.release(7)
        s.run_steps(1, 10)  # the binning leaves at once while the error is not reported
        s.synchronize()
    assert e.value.status == BFVM_ERR_TIMEOUT and "binning" in str(e.value)
    s.synchronize()  # reported once
    s.set_option(option, -1)
    s.set_option("wait_limit_cycles", 4_000_000_000)
    # two steps without secretion, the release, one more
    t = _solver(d, internalized, field, amounts)
    for step in range(3):
        t.diffusion()
        t.gradient()
        if step == 1:
            t.release(7)
    _same(_all(s), _all(t))
    s.run_steps(12, 1)
    t.run_steps(12, 1)
    _same(_all(s), _all(t))
    s.close()
    t.close()


def test_agents_added_before_the_report():
    """The scratch of the grown storage holds no error: the agents are binned and sorted when it is reported."""
    d = _state(3)
    s = _solver(d, True)
    s.set_option("wait_limit_cycles", 2_000_000)
    s.set_option("test_drop_bin_tile", 0)
    s.run_steps(1, 0)
    s.set_option("test_drop_bin_tile", -1)
    rng = np.random.default_rng(1)
    n = 30_000
    more = [rng.random((n, S), dtype=np.float32) for _ in range(6)]
    vol, pos = np.full(n, 1000.0, np.float32), rng.random((n, 3), dtype=np.float32) * np.float32(EDGE * 20 - 1)
    s.add_agents(n, *more, vol, pos)
    s.run_steps(2, 1)
    with pytest.raises(BfvmError) as e:
        s.synchronize()
    assert e.value.status == BFVM_ERR_TIMEOUT
    t = _solver(d, True)
    t.diffusion()
    t.gradient()
    t.add_agents(n, *more, vol, pos)
    t.run_steps(2, 1)
    _same(_all(s), _all(t))
    s.run_steps(3, 3)
    t.run_steps(3, 3)
    _same(_all(s), _all(t))
    s.close()
    t.close()


def test_batch_member_recovers():
    d, other = _state(5), _state(6)
    s, u = _solver(d, True), _solver(other, True)
    b = Batch([s, u])
    b.run_steps(2, 0)
    b.synchronize()
    field, _, amounts = _all(s)
    s.set_option("wait_limit_cycles", 2_000_000)
    s.set_option("test_drop_segment_tile", 3)
    b.run_steps(2, 0)
    with pytest.raises(BfvmError) as e:
        b.synchronize()
    assert e.value.status == BFVM_ERR_TIMEOUT
    s.set_option("test_drop_segment_tile", -1)
    t, v = _solver(d, True, field, amounts), _solver(other, True)
    for _ in range(2):
        t.diffusion()
        t.gradient()
    v.run_steps(2, 0)
    v.run_steps(2, 0)
    b.run_steps(12, 2)
    b.synchronize()
    t.run_steps(12, 2)
    v.run_steps(12, 2)
    _same(_all(s), _all(t))
    _same(_all(u), _all(v))
    b.close()
    for x in (s, u, t, v):
        x.close()


def test_options_are_checked():
    s = _solver(_state(1), True)
    for name in ("test_drop_bin_tile", "test_drop_segment_tile"):
        with pytest.raises(BfvmError):
            s.set_option(name, -2)
    s.close()
