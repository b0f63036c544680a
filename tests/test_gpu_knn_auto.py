"""AUTO's choice between the SIMT kernel and the tensor cores: the same rows on both sides of the line, at the scales
where f32 distances lose digits or leave their range, and for the approximate mode below its own line."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(n, d, seed=0):
    rng = np.random.default_rng(seed)
    return (rng.normal(size=(n, d)) + 4 * rng.normal(size=(12, d))[rng.integers(12, size=n)]).astype(np.float32)


@pytest.mark.parametrize("n,d,k", [(4999, 20, 15), (5000, 20, 15), (5121, 67, 60), (7001, 300, 20), (16383, 12, 30)])
def test_auto_matches_oracle(lib, orc, n, d, k):
    x = _data(n, d, n)
    gi, gd = lib.knn.find_k_nearest_neighbors(x, k)
    rows = np.arange(0, n, 7, dtype=np.uint32)
    ei, ed = orc.knn_rows(x, rows, k)
    assert np.array_equal(gd[rows], ed) and np.array_equal(gi[rows], ei)


@pytest.mark.parametrize("scale", [1e-25, 1e-15, 1e-9, 1e-8, 1e14, 1e16, 1e20])
def test_auto_at_any_scale_matches_simt(lib, scale):
    x = _data(5200, 24, 3) * np.float32(scale)
    gi, gd = lib.knn.find_k_nearest_neighbors(x, 20)
    ei, ed = lib.knn.find_k_nearest_neighbors(x, 20, knn_mode=lib.KnnMode.SIMT_EXACT)
    assert np.array_equal(gd, ed) and np.array_equal(gi, ei)


def test_auto_with_differences_below_the_normal_range(lib):
    """A group of rows whose squared differences are subnormal or vanish, beside rows of ordinary size."""
    rng = np.random.default_rng(1)
    for small in (1e-17, 1e-19, 3e-22, 1e-24):
        x = _data(5300, 16, 5)
        x[100:400] = small * rng.normal(size=(300, 16))
        gi, gd = lib.knn.find_k_nearest_neighbors(x, 25)
        ei, ed = lib.knn.find_k_nearest_neighbors(x, 25, knn_mode=lib.KnnMode.SIMT_EXACT)
        assert np.array_equal(gd, ed) and np.array_equal(gi, ei)


def test_approximate_mode_is_exact_below_its_line(lib):
    x = _data(9000, 30, 8)
    gi, gd = lib.knn.find_k_nearest_neighbors(x, 30, knn_mode=lib.KnnMode.APPROX)
    ei, ed = lib.knn.find_k_nearest_neighbors(x, 30, knn_mode=lib.KnnMode.SIMT_EXACT)
    assert np.array_equal(gd, ed) and np.array_equal(gi, ei)


def test_auto_with_nan_and_inf_rows(lib, orc):
    """A NaN row is nobody's neighbour (the oracle's indices); with an infinite value AUTO is the SIMT kernel."""
    x = _data(5100, 10, 9)
    x[17, 3] = np.nan
    gi, gd = lib.knn.find_k_nearest_neighbors(x, 12)
    ei, ed = orc.knn_exact(x, 12)
    rest = np.arange(len(x)) != 17
    assert np.array_equal(gi, ei) and np.array_equal(gd[rest], ed[rest])
    x[29, 0] = np.inf
    gi, gd = lib.knn.find_k_nearest_neighbors(x, 12)
    ei, ed = lib.knn.find_k_nearest_neighbors(x, 12, knn_mode=lib.KnnMode.SIMT_EXACT)
    assert np.array_equal(gd, ed, equal_nan=True) and np.array_equal(gi, ei)
