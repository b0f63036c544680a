"""The principal axes computed on the device against the host's, bit for bit (both sum in the same order)."""
import numpy as np
import pytest

from pacmap_b200._abi import ptr

pytestmark = pytest.mark.gpu


# 161: the smallest matrix the device takes; 784 x 100: a fit's; 1024 x 128: the largest, 19 columns per block;
# 163 x 2: fewer columns (26) than lanes; rank 40 < k + 24: zero columns after orthonormalisation
@pytest.mark.parametrize("d,k,rank", [(161, 100, 161), (163, 2, 163), (200, 128, 40), (400, 100, 400), (784, 100, 784),
                                      (1024, 128, 1024)])
def test_device_axes_are_the_hosts(lib, d, k, rank):
    rng = np.random.default_rng(d + k)
    f = rng.normal(size=(rank, d)) * np.exp(rng.uniform(-3, 1, size=(rank, 1)))
    cov = np.ascontiguousarray(f.T @ f)
    host = lib.stages.pca_axes(cov, k)
    dev = np.zeros((d, k))
    lib._check(lib._abi.lib().pacmap_pca_axes_device(ptr(cov), d, k, 0, ptr(dev)))
    assert np.array_equal(host, dev)


def test_device_axes_reject_what_they_do_not_take(lib):
    cov = np.eye(160)
    out = np.zeros((160, 2))
    with pytest.raises(lib.Unsupported):
        lib._check(lib._abi.lib().pacmap_pca_axes_device(ptr(cov), 160, 2, 0, ptr(out)))
