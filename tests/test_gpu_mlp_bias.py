"""Bias gradients (column sums staged through shared memory in slices of 256 rows) against the numpy oracle with the
same BF16 rounding points. The tolerance is the one of the whole gradient's test: 0.5 % of the tensor's norm (dZ is
rounded to BF16, 2^-9 relative, on both sides, and a rounding may fall the other way)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
H = 512


# below one slice, exactly one, one and a half, many with a remainder; one output column to a full tile of 16
@pytest.mark.parametrize("batch,dim", [(128, 1), (256, 2), (384, 16), (4224, 3)])
def test_bias_gradients_match_oracle(lib, batch, dim):
    from oracle import mlp as om
    from pacmap_b200 import learned

    rng = np.random.default_rng(batch + dim)
    d = 24
    p = learned.init_params(d, dim, seed=5)
    x = rng.normal(scale=0.7, size=(batch, d)).astype(np.float32)
    t = rng.normal(size=(batch, dim)).astype(np.float32)
    _, g = learned.gradient(p, x, t)
    _, go = om.loss_and_grad(p, x, t, d, dim, bf16_ops=True)
    at = 0
    for size, bias in ((H * d, False), (H, True), (H * H, False), (H, True), (dim * H, False), (dim, True)):
        if bias:
            a, b = g[at:at + size], go[at:at + size]
            assert np.linalg.norm(a - b) <= 5e-3 * np.linalg.norm(b)
        at += size
