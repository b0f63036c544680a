"""The SIMT kNN's staged selection and key slices against the oracle, on every row: list sizes on both sides of each
staging rule, key counts around tiles of 64 and slices of 512, descending distances (every key is a candidate)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k", [(65, 3, 64), (130, 8, 1), (513, 20, 64), (1100, 5, 65), (1025, 16, 192), (2049, 12, 193),
                                   (1500, 9, 448), (4097, 24, 30)])
def test_simt_selection_matches_oracle(lib, orc, n, d, k):
    rng = np.random.default_rng(n + k)
    x = rng.normal(size=(n, d)).astype(np.float32)
    x[::7] = np.round(x[::7])  # ties
    gi, gd = lib.knn.find_k_nearest_neighbors(x, k, knn_mode=lib.KnnMode.SIMT_EXACT)
    ei, ed = orc.knn_exact(x, k)
    assert np.array_equal(gd, ed) and np.array_equal(gi, ei)


def test_simt_selection_with_keys_in_descending_distance(lib, orc):
    n = 3000
    x = (np.arange(n, 0, -1)[:, None] ** 1.5 * np.ones((1, 4))).astype(np.float32)
    gi, gd = lib.knn.find_k_nearest_neighbors(x, 50, knn_mode=lib.KnnMode.SIMT_EXACT)
    ei, ed = orc.knn_exact(x, 50)
    assert np.array_equal(gd, ed) and np.array_equal(gi, ei)
