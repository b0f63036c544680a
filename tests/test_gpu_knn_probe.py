"""The approximate search's rows depend on its pivots' cells, so the choice of pivots is part of its results: checksums of
its neighbours and distances on structureless data, where every cell matters, recorded when the mode was introduced (all
256 pivots by k-means++ draws on at most 65,536 rows). At the first size it takes, at a size that is no multiple of a
block, and with more rows than the subsample holds."""
import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k,idx,dist", [(16384, 24, 15, 0xD5753B20, 0x70C5C6C3), (33000, 40, 30, 0x6895DC57, 0x4851C57C),
                                            (70001, 16, 20, 0xDCF4B84E, 0x120D5B16)])
def test_approximate_rows_stay_the_same(lib, n, d, k, idx, dist):
    x = np.random.default_rng(n).integers(-1000, 1000, size=(n, d)).astype(np.float32)
    gi, gd = lib.knn.find_k_nearest_neighbors(x, k, knn_mode=lib.KnnMode.APPROX)
    assert (zlib.crc32(gi.tobytes()), zlib.crc32(gd.tobytes())) == (idx, dist)
