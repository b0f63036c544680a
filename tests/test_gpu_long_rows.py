"""Points in more than 1,024 pair entries, which the gradient gives a warp instead of eight lanes, against the oracle
(the bounds of the other gradient tests: 1e-5 of a row's sum of |contributions|; Adam bit for bit)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _hubs(n, sizes, seed):
    """Grouped lists in which point h is a partner of about sizes[h] points, split over the three lists; the other
    partners are uniform."""
    rng = np.random.default_rng(seed)
    lists = []
    for k, share in ((10, 0.5), (5, 0.2), (20, 0.3)):
        p = rng.integers(0, n, size=(n, k))
        for h, size in enumerate(sizes):
            rows = rng.choice(np.arange(len(sizes), n), size=min(int(size * share), n - len(sizes)), replace=False)
            p[rows, h % k] = h
        lists.append(np.stack([np.repeat(np.arange(n), k), p.reshape(-1)], 1).astype(np.uint32))
    return lists


# around the rule's 1,024 entries (the uniform partners add ~35 to 70), several rounds of 128, remainders of 32
@pytest.mark.parametrize("dim", [1, 2, 3, 8])
def test_long_rows_match_oracle(lib, orc, dim):
    n = 9000
    pairs = _hubs(n, [900, 960, 1000, 1060, 1500, 2049, 7000], seed=dim)
    y = np.random.default_rng(3).normal(0, 3, size=(n, dim)).astype(np.float32)
    for w in [(2.0, 1000.0, 1.0), (1.0, 0.0, 1.0)]:
        got = lib.stages.gradient(y, *pairs, *w)
        assert np.array_equal(got, lib.stages.gradient(y, *pairs, *w))
        exp, exp64, absum = orc.grad(y, *pairs, *w, with64=True)
        assert (np.abs(got[:-1] - exp64[:-1]) <= TOL * absum + 1e-30).all()
        assert abs(got[-1, 0] - exp64[-1, 0]) <= TOL * abs(exp64[-1, 0])


def test_long_rows_keep_the_order_of_eight_lanes(lib, orc):
    """A long row's sum is the sum that eight lanes form (entry t to lane t % 8, each lane in order, then pairwise
    over lanes 4, 2 and 1 apart), bit for bit; through three optimiser iterations with Adam on the GPU's gradient."""
    n, hub = 4000, 0
    pnn, pmn, pfp = _hubs(n, [3000], seed=5)
    y = np.random.default_rng(4).normal(0, 3, size=(n, 2)).astype(np.float32)
    got = lib.stages.gradient(y, pnn, pmn, pfp, 2.0, 500.0, 1.0)[hub]
    f32 = np.float32
    lanes = np.zeros((8, 2), f32)
    for p, w, c1, c2, sign, whole in ((pnn, 2.0, 10, 20, 1, True), (pmn, 500.0, 10000, 20000, 1, False),
                                      (pfp, 1.0, 1, 2, -1, False)):
        fwd = p[(p[:, 0] == hub) & (p[:, 1] != hub), 1]
        rev = np.sort(p[(p[:, 1] == hub) & (p[:, 0] != hub), 0])
        part = np.sort(np.concatenate([fwd, rev])) if whole else np.concatenate([fwd, rev])
        df = (y[hub] - y[part]).astype(f32)
        dsq = (f32(1) + df[:, 0] * df[:, 0]).astype(f32)
        dsq = (dsq + df[:, 1] * df[:, 1]).astype(f32)
        t = (f32(c1) + dsq).astype(f32)
        w1 = (f32(w) * (f32(c2) / (t * t))).astype(f32)
        term = (w1[:, None] * df).astype(f32) * f32(sign)
        for e in range(part.size):
            lanes[e % 8] += term[e]
    for o in (4, 2, 1):
        lanes = lanes + lanes[np.arange(8) ^ o]
    assert np.array_equal(got, lanes[0])
    m, v = np.zeros_like(y), np.full_like(y, 0.5)
    yg, mg, vg = y.copy(), m.copy(), v.copy()
    g = lib.stages.optimize_steps(yg, mg, vg, pnn, pmn, pfp, 1.0, 100, 100, 150, 151)
    orc.adam(y, g, m, v, 1.0, 150)
    assert np.array_equal(yg, y) and np.array_equal(mg, m) and np.array_equal(vg, v)
