"""Inference around the network: rows preprocessed on the way in (any column count, aligned or not, ragged row counts) and
destandardised on the way out, bit for bit what the separate stages give."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,dim", [(1, 1, 1), (127, 7, 2), (129, 64, 3), (1000, 100, 2), (257, 130, 16), (4096, 128, 2),
                                     (300, 513, 8)])
def test_transform_is_preprocess_apply_destandardise(lib, n, d, dim):
    from pacmap_b200 import learned

    rng = np.random.default_rng(n + d)
    x = rng.normal(1, 2, size=(n, d)).astype(np.float32)
    params = learned.init_params(d, dim, seed=n)
    mean = rng.normal(size=d).astype(np.float32)
    t_mean, t_std = rng.normal(size=dim).astype(np.float32), rng.uniform(1, 5, size=dim).astype(np.float32)
    m = learned.LearnedModel(params, d, dim, -3.5, 9.25, mean, t_mean, t_std)
    xp = ((x - np.float32(-3.5)) / np.float32(9.25) - mean).astype(np.float32)
    want = learned.apply(params, xp, dim) * t_std + t_mean
    assert np.array_equal(m.transform(x), want.astype(np.float32))


def test_apply_in_every_output_column(lib):
    from pacmap_b200 import learned

    rng = np.random.default_rng(2)
    d, dim, n = 77, 5, 333
    p = learned.init_params(d, dim, seed=9)
    x = rng.normal(scale=0.7, size=(n, d)).astype(np.float32)
    got = learned.apply(p, x, dim)
    h = 512
    at = np.cumsum([0, h * d, h, h * h, h, dim * h, dim])
    w1, b1, w2, b2, w3, b3 = (p[a:b].astype(np.float64) for a, b in zip(at[:-1], at[1:]))
    f = np.maximum(x @ w1.reshape(h, d).T + b1, 0)
    f = np.maximum(f @ w2.reshape(h, h).T + b2, 0) @ w3.reshape(dim, h).T + b3
    # BF16 operands in three layers: 2^-9 relative each, as in the existing inference tests
    assert np.linalg.norm(got - f) <= 2e-2 * np.linalg.norm(f)
