"""The optimiser that keeps every row resident for all iterations against the one with a launch per iteration (asking
for the losses takes the latter): y and the snapshots bit for bit, at one block, many, the last sizes that fit and the
first that do not, in every embedding dimension, with all phases, odd iteration counts and snapshots in each phase."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _both(lib, x, cfg):
    a, sa = lib.fit_transform(x, cfg)
    b, sb, _ = lib.fit_transform(x, cfg, loss_trace=True)
    assert np.array_equal(a, b)
    assert (sa is None and sb is None) or np.array_equal(sa, sb)
    assert np.isfinite(a).all()


@pytest.mark.parametrize("n", [2, 31, 32, 33, 700, 4737, 9473, 14208, 14209, 18944, 18945])
def test_resident_equals_one_launch_per_iteration(lib, n):
    x = np.random.default_rng(n).normal(size=(n, 12)).astype(np.float32)
    cfg = lib.Configuration(initialization=lib.Initialization.Random(3), seed=5, num_iters=(4, 3, 6),
                            far_pair_ratio=1.0 if n < 100 else 2.0, override_neighbors=1 if n < 100 else None,
                            mid_near_ratio=0.0 if n < 100 else 0.5)
    _both(lib, x, cfg)


@pytest.mark.parametrize("dim", [1, 2, 3, 4, 5, 6, 7, 8])
def test_resident_dimensions_and_snapshots(lib, dim):
    x = np.random.default_rng(dim).normal(size=(1500, 20)).astype(np.float32)
    cfg = lib.Configuration(initialization=lib.Initialization.Random(3), seed=5, num_iters=(5, 4, 4), embedding_dimensions=dim,
                            snapshots=[0, 2, 7, 7, 13, 99])
    _both(lib, x, cfg)
    _both(lib, x, dataclasses.replace(cfg, num_iters=(0, 0, 1), snapshots=None))
