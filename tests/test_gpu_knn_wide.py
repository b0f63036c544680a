"""Rows whose candidate band overflows the filter's buffer and that are settled over column lists: indices and f32
distances equal to the exact SIMT kernel's on every row (it forms every distance in the reference's order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _near_duplicates(n, d, dups, seed):
    """A far-off mixture in which `dups` rows coincide and as many lie within a tiny distance of them: their distances
    are far below the filter's error bound, which scales with the norms."""
    rng = np.random.default_rng(seed)
    x = rng.normal(0, 1, size=(n, d)) + 10 * rng.normal(size=(8, d))[rng.integers(8, size=n)]
    at = rng.permutation(n)
    x[at[:dups]] = x[at[0]]
    x[at[dups:2 * dups]] = x[at[0]] + 1e-4 * rng.normal(size=(dups, d))
    return x.astype(np.float32)


# every operand staging (1, 2, 3, 4 and more blocks of 64 columns), remainders of 8 columns, both buffer sizes
# (k = 250), both operand types; row counts off the 128 and 256 tiles; one row block (its column tiles split over the
# SMs) to 40 of them
@pytest.mark.parametrize("n,d,dups,k,mode", [(3001, 24, 600, 60, 1), (4000, 100, 700, 15, 1), (2500, 131, 900, 90, 2),
                                             (3000, 256, 600, 60, 1), (2111, 300, 500, 72, 1), (4099, 64, 1500, 250, 1),
                                             (16500, 40, 5000, 30, 1)])
def test_wide_rows_equal_simt(lib, n, d, dups, k, mode):
    x = _near_duplicates(n, d, dups, seed=n)
    gi, gd = lib.knn.find_k_nearest_neighbors(x, k, knn_mode=mode)
    ei, ed = lib.knn.find_k_nearest_neighbors(x, k, knn_mode=lib.KnnMode.SIMT_EXACT)
    assert np.array_equal(gd, ed) and np.array_equal(gi, ei)


def test_wide_rows_with_pruning_and_shards(lib):
    """Overflow in the bound pass of the tile pruning, and rows split over shards, against SIMT."""
    x = _near_duplicates(34000, 48, 3000, seed=2)
    ei, ed = lib.knn.find_k_nearest_neighbors(x, 40, knn_mode=lib.KnnMode.SIMT_EXACT)
    gi, gd = lib.knn.find_k_nearest_neighbors(x, 40)
    assert np.array_equal(gd, ed) and np.array_equal(gi, ei)
    seen = np.zeros(len(x), int)
    for shard in range(3):
        si, sd, own = lib.knn.find_k_nearest_neighbors_shard(x, 40, shard, 3)
        assert np.array_equal(si[own], ei[own]) and np.array_equal(sd[own], ed[own])
        seen += own
    assert (seen == 1).all()


def test_wide_rows_settle_image_like_data(lib):
    """Image-like rows (many near-black images): no row is left to the SIMT kernel over all columns."""
    from pacmap_b200 import datasets

    x, _ = datasets.image_like(n=20000, d=784, seed=5)
    lib.set_stage_timing(True)
    try:
        lib.fit_transform(x, lib.Configuration(seed=3, initialization=lib.Initialization.Random(1), num_iters=(0, 0, 1)))
        st = lib.stage_times()
    finally:
        lib.set_stage_timing(False)
    assert st["knn_fallback_rows"] == 0, st
