"""The one-block Jacobi of small covariances against numpy's f64 eigh, and the matrices it leaves to the host."""
import ctypes as C

import numpy as np
import pytest

from pacmap_b200._abi import ptr

pytestmark = pytest.mark.gpu


def axes(lib, cov, k):
    cov = np.ascontiguousarray(cov, np.float64)
    out, found = np.full((cov.shape[0], k), -7.0), C.c_int32(-1)
    lib._check(lib._abi.lib().pacmap_debug_small_axes(ptr(cov), cov.shape[0], k, 0, ptr(out), C.byref(found)))
    return out, found.value


# 2, 3: the smallest even and odd orders; 31..33: about the line from which fits use it; 65: one block of pairs per
# thread and a few threads with two; 100 x 2: a fit's; 159, 160: the largest; k = 8: the most vectors
@pytest.mark.parametrize("d,k", [(2, 2), (3, 1), (31, 8), (32, 2), (33, 3), (65, 8), (100, 2), (159, 8), (160, 8)])
def test_axes_match_eigh(lib, d, k):
    rng = np.random.default_rng(100 * d + k)
    q, _ = np.linalg.qr(rng.normal(size=(d, d)))
    lam = np.concatenate([5.0 * 0.9 ** np.arange(k), 5.0 * 0.9**k * np.sort(rng.uniform(0, 0.9, size=d - k))[::-1]])
    cov = (q * lam) @ q.T
    cov = 0.5 * (cov + cov.T)
    got, found = axes(lib, cov, k)
    assert found == 1
    w, v = np.linalg.eigh(cov)
    v = v[:, ::-1][:, :k]
    v = v * np.sign(v[np.abs(v).argmax(0), np.arange(k)])
    # either method's error is at most about d eps |A| / gap (Davis, Kahan); the gaps here are above 0.04 |A|
    assert np.abs(got - v).max() <= 2 * d * np.finfo(float).eps / 0.04
    assert np.abs(got - lib.stages.pca_axes(cov, k)).max() <= 2 * d * np.finfo(float).eps / 0.04


@pytest.mark.parametrize("case", ["equal", "close", "zero", "rank", "nan", "inf"])
def test_left_to_the_host(lib, case):
    d, k = 40, 2
    rng = np.random.default_rng(3)
    q, _ = np.linalg.qr(rng.normal(size=(d, d)))
    lam = 3.0 * 0.8 ** np.arange(d)
    lam[1:3] = {"equal": (1.0, 1.0), "close": (1.0, 1.0 - 0.0015), "rank": (0.0, 0.0)}.get(case, lam[1:3])
    lam[3:] *= {"rank": 0.0}.get(case, 0.3)
    cov = (q * lam) @ q.T
    if case == "zero":
        cov[:] = 0.0
    if case in ("nan", "inf"):
        cov[5, 5] = np.nan if case == "nan" else np.inf
    got, found = axes(lib, cov, k)
    assert found == 0 and (got == -7.0).all()


def test_rejects_what_it_does_not_take(lib):
    for d, k in [(161, 2), (100, 9), (1, 1), (4, 5)]:
        with pytest.raises(lib.Unsupported):
            axes(lib, np.eye(d), k)
