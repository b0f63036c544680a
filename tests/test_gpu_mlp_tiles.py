"""The network's GEMM tiles: a row's values do not depend on which tile width the call's row count picks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 148 SMs, 512 hidden units: up to 9 row blocks of 128 go through 32-column tiles, 10 and more through 128-column ones
# (six stages up to 37 row blocks, two above)
@pytest.mark.parametrize("d,dim", [(33, 2), (128, 3), (200, 16)])
def test_rows_do_not_depend_on_the_tile(lib, d, dim):
    from pacmap_b200 import learned

    rng = np.random.default_rng(d)
    x = rng.normal(size=(5000, d)).astype(np.float32)
    params = learned.init_params(d, dim, seed=3)
    want = learned.apply(params, x, dim)
    assert np.isfinite(want).all() and np.abs(want).max() > 0
    for n in (1, 128, 129, 1152, 1153, 4736, 4737):
        assert np.array_equal(learned.apply(params, x[:n], dim), want[:n])
