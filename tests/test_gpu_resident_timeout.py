"""Failure detection without a GPU fault: with the test hook on, the resident optimiser's blocks wait for one that does
not exist; the bounded wait runs out, the call fails with a status, and the next call on the same context is right."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [30, 3000])
def test_grid_barrier_runs_out_with_a_status(lib, n):
    rng = np.random.default_rng(n)
    y0 = rng.normal(size=(n, 2)).astype(np.float32)
    pairs = [np.stack([np.repeat(np.arange(n), 4), rng.integers(0, n, 4 * n)], 1).astype(np.uint32) for _ in range(3)]

    def steps():
        y, m, v = y0.copy(), np.zeros_like(y0), np.zeros_like(y0)
        lib.stages.optimize_steps(y, m, v, *pairs, 1.0, 100, 100, 90, 95, want_grad=False)
        return y, m, v

    before = steps()
    stall = lib._abi.lib().pacmap_debug_stall_optimizer
    stall(1)
    try:
        with pytest.raises(lib.DeviceInvariant) as e:
            steps()
        assert "timed out" in str(e.value)
    finally:
        stall(0)
    assert all(np.array_equal(a, b) for a, b in zip(before, steps()))
