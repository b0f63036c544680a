"""Covariance tiles and projection widths of the Pca start, through a fit of no iterations, against numpy in f64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# columns: 16-wide tiles (15, 16, 17, 64, 100) and 64-wide ones (16,500 x 784: 91 tile pairs x 2 row chunks); axes:
# both ends of each projection width (at most 8 up to 100 columns, min(100, rows) = 32 | 33, 64 | 65, 100 above);
# rows: a slab and one more, three row chunks
@pytest.mark.parametrize("n,d,dim", [(33, 15, 2), (300, 16, 3), (700, 17, 8), (1000, 64, 1), (500, 100, 8), (40000, 50, 2),
                                     (32, 130, 2), (33, 130, 3), (64, 150, 2), (65, 150, 2), (2000, 161, 8),
                                     (16500, 784, 2)])
def test_start_is_the_projection(lib, n, d, dim):
    rng = np.random.default_rng(n + d)
    # variances that fall by a fifth per column, then stay: the leading axes are well apart
    scale = np.maximum(0.9 ** np.arange(d), 0.9 ** (dim + 3) * 0.3)
    x = (rng.normal(size=(n, d)) * scale + rng.normal(size=d)).astype(np.float32)
    cfg = lib.Configuration(seed=3, num_iters=(0, 0, 0), embedding_dimensions=dim)
    y = lib.fit_transform(x, cfg)[0]
    z = (lib.stages.preprocess(x)[0] if d <= 100 else x).astype(np.float64)
    zc = z - z.mean(0)
    w, v = np.linalg.eigh(zc.T @ zc)
    v = v[:, ::-1][:, :dim]
    v = v * np.sign(v[np.abs(v).argmax(0), np.arange(dim)])
    # the centred row and the axis are rounded to f32 (2^-24 of each term, |axis| = 1), then the result, and the wide
    # data's column is scaled after its own rounding
    tol = 0.01 * (2 * 2.0**-24 * np.linalg.norm(zc, axis=1, keepdims=True) + 3 * 2.0**-24 * np.abs(zc @ v))
    axis = d * np.finfo(float).eps * w[-1] / np.min(np.diff(w[::-1][:dim + 1]) * -1)  # f64 rounding, both sides
    tol = tol + 0.01 * 2 * axis * np.linalg.norm(zc, axis=1, keepdims=True)
    assert (np.abs(y - 0.01 * (zc @ v)) <= tol).all()
