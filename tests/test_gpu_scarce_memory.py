"""Calls that get no memory beyond what they cannot do without: the same results, by the slower way. (The allocations are
refused on the host by a hook of the calling thread.)"""
import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def _scarce(lib):
    hook = lib._abi.lib().pacmap_debug_scarce_memory
    hook(1)
    try:
        yield
    finally:
        hook(0)


def test_copies_without_page_locked_slots(lib, orc):
    """42 MB up and down, past the sizes from which copies are staged."""
    x = np.random.default_rng(0).uniform(-2, 3, size=(105001, 100)).astype(np.float32)
    with _scarce(lib):
        got = lib.stages.preprocess(x)[0]
    assert np.array_equal(got, orc.preprocess(x)[0])
    assert np.array_equal(lib.stages.preprocess(x)[0], got)


def test_gradient_without_tile_lists(lib):
    """66,001 points in 3-D: the row-by-row gradient's bits, and a fit that goes through."""
    n = 66001
    rng = np.random.default_rng(0)
    pairs = [np.stack([np.repeat(np.arange(n), k), rng.integers(0, n, n * k)], 1).astype(np.uint32) for k in (12, 6, 24)]
    y = rng.normal(0, 4, size=(n, 3)).astype(np.float32)
    cfg = lib.Configuration(initialization=lib.Initialization.Random(3), seed=5, num_iters=(4, 4, 4), embedding_dimensions=3,
                            pair_configuration=lib.PairConfiguration.AllProvided(*pairs))
    with _scarce(lib):
        g = lib.stages.optimize_steps(y.copy(), np.zeros_like(y), np.zeros_like(y), *pairs, 1.0, 100, 100, 150, 151)
        e, _ = lib.fit_transform(y, cfg)
    assert np.array_equal(g, lib.stages.gradient(y, *pairs, 3.0, 3.0, 1.0))
    a, _ = lib.fit_transform(y, cfg)
    assert np.linalg.norm(a - e) <= 1e-4 * np.linalg.norm(a) and not np.array_equal(a, e)


def test_knn_below_16384_rows_without_filter_buffers(lib):
    x = np.random.default_rng(1).normal(size=(6001, 20)).astype(np.float32)
    with _scarce(lib):
        gi, gd = lib.knn.find_k_nearest_neighbors(x, 15)
    ei, ed = lib.knn.find_k_nearest_neighbors(x, 15)
    assert np.array_equal(gi, ei) and np.array_equal(gd, ed)


def test_knn_of_overflowed_rows_without_column_lists(lib, orc):
    """2,000 exact ties and a dense clump far from the origin, more than the filter's buffers hold."""
    rng = np.random.default_rng(2)
    x = rng.normal(size=(17001, 24)).astype(np.float32)
    x[3000:5000] = x[3000]
    x[9000:12000] = 300 + 0.001 * rng.normal(size=(3000, 24)).astype(np.float32)
    with _scarce(lib):
        gi, gd = lib.knn.find_k_nearest_neighbors(x, 20)
    ei, ed = lib.knn.find_k_nearest_neighbors(x, 20)
    assert np.array_equal(gi, ei) and np.array_equal(gd, ed)
    rows = np.arange(0, 17001, 29, dtype=np.uint32)
    oi, od = orc.knn_rows(x, rows, 20)
    assert np.array_equal(gi[rows], oi) and np.array_equal(gd[rows], od)
