"""The launch count names launches that were made."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_gradient_counts_the_long_rows_kernel_only_when_it_runs(lib):
    """The same lists but for one point, whose 3 x 400 entries in the second make it a row of more than 1,024 (in segments
    that the list building treats like the others): one launch more."""
    n = 3000
    rng = np.random.default_rng(0)
    y = rng.normal(size=(n, 2)).astype(np.float32)
    pairs = [np.stack([np.repeat(np.arange(n), 4), rng.integers(0, n, 4 * n)], 1).astype(np.uint32) for _ in range(3)]
    counts = []
    for hub in (False, True):
        if hub:
            for p in pairs:
                p[rng.choice(4 * n, 400, replace=False), 1] = 7
        lib.last_launch_count()
        lib.stages.gradient(y, *pairs, 2.0, 500.0, 1.0)
        counts.append(lib.last_launch_count())
    assert counts[1] == counts[0] + 1
