"""Rows that lie apart from their cell (tile pruning with 1,024 column tiles and more): the pruned search equals the full
sweep on every row, with single far points, small far groups, groups of two densities in one place, and far duplicates."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(n, d, seed):
    rng = np.random.default_rng(seed)
    x = 6 * rng.normal(size=(60, d))[rng.integers(60, size=n)] + rng.normal(size=(n, d))
    at = rng.permutation(n)
    x[at[:150]] += 25 * rng.normal(size=(150, d))                                   # single points
    x[at[150:450]] = 40 * rng.normal(size=(60, d))[np.arange(300) // 5] + 0.1 * rng.normal(size=(300, d))
    x[at[450:20450]] = x[at[450]] + np.where(np.arange(20000) % 2, 0.3, 3.0)[:, None] * rng.normal(size=(20000, d))
    x[at[20450:21450]] = 30 * rng.normal(size=d)                                    # a thousand coincident points
    return x.astype(np.float32)


@pytest.mark.parametrize("n,d,k,mode", [(131073, 24, 40, 0), (140001, 70, 15, 0), (132000, 32, 200, 2)])
def test_pruned_search_with_far_rows_equals_full_sweep(lib, n, d, k, mode):
    x = _data(n, d, n)
    gi, gd = lib.knn.find_k_nearest_neighbors(x, k, knn_mode=mode)
    fi, fd = lib.knn.find_k_nearest_neighbors(x, k, knn_mode=lib.KnnMode.TENSOR_F16_FULL)
    assert np.array_equal(gd, fd) and np.array_equal(gi, fi)


def test_far_rows_in_shards(lib):
    x = _data(131200, 20, 3)
    ei, ed = lib.knn.find_k_nearest_neighbors(x, 20)
    seen = np.zeros(len(x), int)
    for shard in range(2):
        si, sd, own = lib.knn.find_k_nearest_neighbors_shard(x, 20, shard, 2)
        assert np.array_equal(si[own], ei[own]) and np.array_equal(sd[own], ed[own])
        seen += own
    assert (seen == 1).all()
